// What the gpt-oss attention kernels share: the operands of one call and the addressing of the paged cache.
#pragma once
#include "common.cuh"

namespace gb200 {

struct OssAttn {
    const float* qkv;             // [batch * tokens, (q + 2 kv) * d], already rotated
    __nv_bfloat16* keys;          // [layers][physical pages][page size][kv heads][d]
    __nv_bfloat16* values;
    const int* table;             // [batch, logical pages]
    const int* lengths;           // [batch]: positions visible at decode
    const int* starts;            // [batch]: position of the first new token
    const int* active;            // [batch]
    const float* sinks;           // [q heads]
    float* out;                   // [batch * tokens, q * d]
    int batch, tokens, logical_pages, physical_pages;
    int q_heads, kv_heads, head_dim, layer, page_size, window, prefill;
};

#if defined(__CUDACC__)
__device__ __forceinline__ size_t oss_cache_offset(const OssAttn& p, int b, int position, int head)
{
    if (position < 0 || position / p.page_size >= p.logical_pages) return SIZE_MAX;
    const int page = p.table[b * p.logical_pages + position / p.page_size];
    if (page < 0 || page >= p.physical_pages) return SIZE_MAX;
    return (((size_t(p.layer) * p.physical_pages + page) * p.page_size + position % p.page_size) * p.kv_heads + head) * p.head_dim;
}

// One row of the output, any head size up to 256, one warp: online softmax in position order, the sink in the denominator only.
__device__ __forceinline__ void oss_attention_row(const OssAttn& p, int row, int head, int lane)
{
    const int b = row / p.tokens, t = row % p.tokens;
    const int packed = (p.q_heads + 2 * p.kv_heads) * p.head_dim;
    float accum[8] = {};
    const int end = p.prefill ? p.starts[b] + t + 1 : p.lengths[b];
    const int begin = p.window ? max(0, end - p.window) : 0;
    float maximum = p.sinks[head], sum = 1;
    const float* q = p.qkv + size_t(row) * packed + head * p.head_dim;
    if (p.active[b] && end > 0 && end <= p.logical_pages * p.page_size) {
        for (int pos = begin; pos < end; ++pos) {
            const size_t off = oss_cache_offset(p, b, pos, head / (p.q_heads / p.kv_heads));
            if (off == SIZE_MAX) continue;
            float score = 0;
            for (int d = lane; d < p.head_dim; d += 32) score += q[d] * __bfloat162float(p.keys[off + d]);
#pragma unroll
            for (int o = 16; o; o >>= 1) score += __shfl_xor_sync(0xffffffffu, score, o);
            score *= rsqrtf(float(p.head_dim));
            const float next = fmaxf(maximum, score);
            const float old = expf(maximum - next), weight = expf(score - next);
            sum = sum * old + weight;
            for (int d = lane, i = 0; d < p.head_dim; d += 32, ++i) accum[i] = accum[i] * old + weight * __bfloat162float(p.values[off + d]);
            maximum = next;
        }
    }
    for (int d = lane, i = 0; d < p.head_dim; d += 32, ++i)
        p.out[size_t(row) * p.q_heads * p.head_dim + head * p.head_dim + d] = bf16_round_f(accum[i] / sum);
}

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(valid ? 16 : 0) : "memory");
}
__device__ __forceinline__ uint32_t bf16x2_of(float lo, float hi)
{
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
#endif

// gpt_oss_prefill.cu: many query rows of 64-wide heads on the tensor cores.  `oss_prefill_takes` says whether the shape and
// the alignment of the operands suit it.
constexpr int kOssDim = 64;
bool oss_prefill_takes(const OssAttn& p);
int oss_prefill_launch(const OssAttn& p, cudaStream_t stream);
// gpt_oss_decode.cu: one new token per sequence, 64-wide heads, up to 16 q heads per kv head.
bool oss_decode_takes(const OssAttn& p);
int oss_decode_launch(const OssAttn& p, cudaStream_t stream);

}  // namespace gb200
