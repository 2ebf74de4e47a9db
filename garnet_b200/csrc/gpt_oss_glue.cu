// The rest of a gpt-oss decoder layer around the MoE operator: RMS norm, YaRN rotary
// embedding, paged-KV attention with learned sinks and a sliding window, the bf16 GEMV of the
// q/k/v and output projections at decode, and the per-rank (score, token) pair of the sharded
// vocabulary.  x and y use the reference's fp32 carrier (fp32 tensors that hold bf16 values).
//
// Reference (plugins/gpt_oss/cuda/gpt_oss_kernels.cu): rmsNorm :22-48, rope :78-99,
// cacheOffset / writeKV :100-123, attention :125-160 (one warp per query head, the sink enters the
// softmax denominator only), decodeAttentionPartial / Merge :376-428,:513-535, vocabTop1 :430-455,
// the entry points RunGptOssRmsNorm / Rope / Attention / VocabTop1 :930-1210; decodeGemv
// (plugins/gpt_oss/cuda/gpt_oss_gemv.cu:7-39).
// Attention itself: gpt_oss_decode.cu (one token per sequence), gpt_oss_prefill.cu (many rows) and, for other shapes, the
// row loop here.
#include <cfloat>
#include <cstdint>

#include "gpt_oss_attn.cuh"

namespace gb200 {

namespace {

__device__ __forceinline__ float bfr(float f) { return __bfloat162float(__float2bfloat16_rn(f)); }
__device__ __forceinline__ float warp_sum(float v)
{
#pragma unroll
    for (int off = 16; off; off >>= 1) v += __shfl_xor_sync(0xffffffffu, v, off);
    return v;
}
// y = bf((bf(x) * rsqrt(mean(bf(x)^2) + eps)) * w), one CTA per row.
__global__ void __launch_bounds__(256) oss_rms_norm_kernel(const float* __restrict__ x, const float* __restrict__ w, float* __restrict__ y,
                                                           int hidden, float eps)
{
    __shared__ float part[8];
    const float* xr = x + size_t(blockIdx.x) * hidden;
    float sum = 0.f;
    for (int d = threadIdx.x; d < hidden; d += 256) {
        const float v = bfr(xr[d]);
        sum += v * v;
    }
    sum = warp_sum(sum);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = sum;
    __syncthreads();
    float total = 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) total += part[i];
    const float inv = rsqrtf(total / hidden + eps);
    for (int d = threadIdx.x; d < hidden; d += 256) y[size_t(blockIdx.x) * hidden + d] = bfr((bfr(xr[d]) * inv) * w[d]);
}

struct OssRope {
    int q_heads, kv_heads, head_dim;
    float theta, factor, initial_context, beta_fast, beta_slow;
};

// A CTA rotates two tokens (or a share of one token's heads, when there are few): one thread per (token, frequency)
// computes the angle's powf, logf, cosf and sinf - some hundreds of instructions - once for all heads, then every thread moves
// kVec neighbouring frequencies of a head (16-byte loads and stores when the head size and the pointers allow it).
// Bound: HBM, 2 x 4 bytes per value.  2048 tokens of 64 / 8 heads of 64 (84 MB): 24.0 -> 19.3 us (ncu) against one
// thread per (token, frequency) and eight walking over the heads with 4-byte accesses.
constexpr int kRopeTokens = 2, kRopeThreads = 256, kRopeMaxHalf = 128;

template <int kVec, int kUnroll>
__global__ void __launch_bounds__(kRopeThreads) oss_rope_kernel(const float* __restrict__ x, const long long* __restrict__ positions,
                                                                float* __restrict__ y, int tokens, int per_cta, OssRope o)
{
    __shared__ __align__(16) float cosines[kRopeTokens][kRopeMaxHalf], sines[kRopeTokens][kRopeMaxHalf];
    const int half = o.head_dim / 2, rot_heads = o.q_heads + o.kv_heads;
    const int packed = (o.q_heads + 2 * o.kv_heads) * o.head_dim;
    const int token0 = blockIdx.x * per_cta, count = min(per_cta, tokens - token0);
    pdl_launch_dependents();
    pdl_wait();
    for (int i = threadIdx.x; i < count * half; i += kRopeThreads) {
        const int token = i / half, frequency = i % half;
        const float pi = 3.14159265358979323846f;
        float inv = powf(o.theta, -2.f * frequency / o.head_dim), concentration = 1;
        if (o.factor > 1) {
            const float low = half * logf(o.initial_context / (o.beta_fast * 2 * pi)) / logf(o.theta);
            const float high = half * logf(o.initial_context / (o.beta_slow * 2 * pi)) / logf(o.theta);
            const float ramp = fminf(1, fmaxf(0, (frequency - low) / (high - low)));
            inv *= (1 - ramp) + ramp / o.factor;
            concentration = 1 + .1f * logf(o.factor);
        }
        const float angle = float(positions[token0 + token]) * inv;
        cosines[token][frequency] = bfr(cosf(angle) * concentration);
        sines[token][frequency] = bfr(sinf(angle) * concentration);
    }
    __syncthreads();
    const int pieces = half / kVec, part = blockIdx.y * kRopeThreads + threadIdx.x, parts = gridDim.y * kRopeThreads;
    const int v0 = rot_heads * o.head_dim;
    for (int token = 0; token < count; ++token) {
        const float* xr = x + size_t(token0 + token) * packed;
        float* yr = y + size_t(token0 + token) * packed;
#pragma unroll kUnroll
        for (int i = part; i < rot_heads * pieces; i += parts) {
            const int f = i % pieces * kVec, at = i / pieces * o.head_dim + f;
            float a[kVec], b[kVec], ra[kVec], rb[kVec];
            if constexpr (kVec == 4) {
                *reinterpret_cast<float4*>(a) = __ldg(reinterpret_cast<const float4*>(xr + at));
                *reinterpret_cast<float4*>(b) = __ldg(reinterpret_cast<const float4*>(xr + at + half));
            } else {
                a[0] = xr[at], b[0] = xr[at + half];
            }
#pragma unroll
            for (int j = 0; j < kVec; ++j) {
                const float cosine = cosines[token][f + j], sine = sines[token][f + j];
                ra[j] = bfr(bfr(a[j] * cosine) + bfr(-b[j] * sine));
                rb[j] = bfr(bfr(b[j] * cosine) + bfr(a[j] * sine));
            }
            if constexpr (kVec == 4) {
                *reinterpret_cast<float4*>(yr + at) = *reinterpret_cast<const float4*>(ra);
                *reinterpret_cast<float4*>(yr + at + half) = *reinterpret_cast<const float4*>(rb);
            } else {
                yr[at] = ra[0], yr[at + half] = rb[0];
            }
        }
        // the v part passes through
        for (int c = v0 + part * kVec; c < packed; c += parts * kVec) {
            if constexpr (kVec == 4) *reinterpret_cast<float4*>(yr + c) = __ldg(reinterpret_cast<const float4*>(xr + c));
            else yr[c] = xr[c];
        }
    }
}

// Appends the rows' k and v at positions starts[b] + t.  A thread takes kVec neighbouring values of k or v (8 when the head
// size and the pointers allow it): one page lookup and one 16-byte store for eight of them.
template <int kVec>
__global__ void oss_write_kv_kernel(const OssAttn p)
{
    const int kv_width = p.kv_heads * p.head_dim, packed = (p.q_heads + 2 * p.kv_heads) * p.head_dim, pieces = 2 * kv_width / kVec;
    const size_t idx = size_t(blockIdx.x) * blockDim.x + threadIdx.x;
    pdl_launch_dependents();
    pdl_wait();
    if (idx >= size_t(p.batch) * p.tokens * pieces) return;
    const int row = int(idx / pieces), b = row / p.tokens, t = row % p.tokens, c = int(idx % pieces) * kVec, is_v = c >= kv_width;
    const int d = is_v ? c - kv_width : c;
    if (!p.active[b]) return;
    const size_t off = oss_cache_offset(p, b, p.starts[b] + t, d / p.head_dim);
    if (off == SIZE_MAX) return;
    const float* src = p.qkv + size_t(row) * packed + p.q_heads * p.head_dim + c;
    __nv_bfloat16* dst = (is_v ? p.values : p.keys) + off + d % p.head_dim;
    if constexpr (kVec == 8) {
        const float4 lo = __ldg(reinterpret_cast<const float4*>(src)), hi = __ldg(reinterpret_cast<const float4*>(src) + 1);
        const __nv_bfloat162 v[4] = {__floats2bfloat162_rn(lo.x, lo.y), __floats2bfloat162_rn(lo.z, lo.w),
                                     __floats2bfloat162_rn(hi.x, hi.y), __floats2bfloat162_rn(hi.z, hi.w)};
        *reinterpret_cast<uint4*>(dst) = *reinterpret_cast<const uint4*>(v);
    } else {
        *dst = __float2bfloat16(*src);
    }
}

// Any shape: one warp per (row, q head), online softmax in position order (the reference's baseline).
__global__ void oss_attention_generic_kernel(const OssAttn p)
{
    const int task = int((size_t(blockIdx.x) * blockDim.x + threadIdx.x) / 32);
    if (task >= p.batch * p.tokens * p.q_heads) return;
    oss_attention_row(p, task / p.q_heads, task % p.q_heads, threadIdx.x & 31);
}

__global__ void __launch_bounds__(256) oss_vocab_top1_kernel(const float* __restrict__ logits, float* __restrict__ pairs, int width, int rank)
{
    __shared__ float s_val[8];
    __shared__ int s_idx[8];
    const float* row = logits + size_t(blockIdx.x) * width;
    float best = -FLT_MAX;
    int arg = 0;
    for (int i = threadIdx.x; i < width; i += 256) {
        const float v = row[i];
        if (v > best || (v == best && i < arg)) best = v, arg = i;
    }
#pragma unroll
    for (int off = 16; off; off >>= 1) {
        const float ov = __shfl_xor_sync(0xffffffffu, best, off);
        const int oa = __shfl_xor_sync(0xffffffffu, arg, off);
        if (ov > best || (ov == best && oa < arg)) best = ov, arg = oa;
    }
    if ((threadIdx.x & 31) == 0) s_val[threadIdx.x >> 5] = best, s_idx[threadIdx.x >> 5] = arg;
    __syncthreads();
    if (threadIdx.x == 0) {
        for (int i = 1; i < 8; ++i)
            if (s_val[i] > best || (s_val[i] == best && s_idx[i] < arg)) best = s_val[i], arg = s_idx[i];
        pairs[size_t(blockIdx.x) * 2] = best;
        pairs[size_t(blockIdx.x) * 2 + 1] = float(rank * width + arg);
    }
}

// y[row] = bf16(sum_c w[weight_row(row), offset + c] * x[c]); one warp per row, 16-byte loads.
__global__ void __launch_bounds__(128) oss_gemv_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w,
                                                       __nv_bfloat16* __restrict__ y, int rows, int columns, int stride, int offset,
                                                       int q_heads, int kv_heads, int head_dim, int rank)
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int row = blockIdx.x * 4 + warp;
    if (row >= rows) return;
    int wr = row;
    if (q_heads > 0) {   // this rank's half of the q, k and v rows of a packed q/k/v weight
        const int qp = (q_heads / 2) * head_dim, kp = (kv_heads / 2) * head_dim;
        wr = row < qp ? rank * qp + row : row < qp + kp ? q_heads * head_dim + rank * kp + row - qp : (q_heads + kv_heads) * head_dim + rank * kp + row - qp - kp;
    }
    const __nv_bfloat16* v = w + size_t(wr) * stride + offset;
    float sum = 0.f;
    if ((((reinterpret_cast<uintptr_t>(v) | reinterpret_cast<uintptr_t>(x)) & 15) == 0) && columns % 8 == 0) {
        for (int c = lane * 8; c < columns; c += 256) {
            const uint4 a = __ldg(reinterpret_cast<const uint4*>(v + c)), bx = __ldg(reinterpret_cast<const uint4*>(x + c));
            const uint32_t aw[4] = {a.x, a.y, a.z, a.w}, bw[4] = {bx.x, bx.y, bx.z, bx.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sum = fmaf(__uint_as_float(aw[i] << 16), __uint_as_float(bw[i] << 16), sum);
                sum = fmaf(__uint_as_float(aw[i] & 0xffff0000u), __uint_as_float(bw[i] & 0xffff0000u), sum);
            }
        }
    } else {
        for (int c = lane; c < columns; c += 32) sum = fmaf(__bfloat162float(v[c]), __bfloat162float(x[c]), sum);
    }
    sum = warp_sum(sum);
    if (lane == 0) y[row] = __float2bfloat16_rn(sum);
}

int validate_oss(const garnet_b200_gpt_oss_options* o, bool attention)
{
    if (!o) return fail(GARNET_B200_INVALID_VALUE, "gpt_oss: null options");
    if (o->abi != GARNET_B200_ABI || o->struct_size != int(sizeof(garnet_b200_gpt_oss_options)))
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss: options abi/size mismatch (abi %d, size %d)", o->abi, o->struct_size);
    if (o->q_heads <= 0 || o->kv_heads <= 0 || o->q_heads % o->kv_heads || o->head_dim <= 0 || o->head_dim % 2 || o->head_dim > 256)
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss: bad head geometry");
    if (attention && (o->page_size <= 0 || o->layer < 0 || o->window < 0))
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss: page_size must be positive, layer and window non-negative");
    return GARNET_B200_OK;
}

// The workspace that a decode call brings: a counter per (sequence, kv head) and a record of 2 + 64 numbers per (q head, 64
// positions).  The size is part of the interface; the decode kernel merges its splits on the chip and leaves it alone.
size_t oss_workspace(const garnet_b200_gpt_oss_options& o, int batch, int logical_pages)
{
    const int span = o.window ? std::min(o.window, logical_pages * o.page_size) : logical_pages * o.page_size;
    const int splits = std::max(1, (span + 63) / 64);
    const size_t counters = (size_t(batch) * o.kv_heads * 4 + 255) & ~size_t(255);
    return counters + size_t(batch) * o.q_heads * splits * (2 + kOssDim) * 4;
}

// A launch that may start while the kernel before it drains (its griddepcontrol.wait is where it waits for that kernel).
template <typename... Params, typename... Args>
cudaError_t launch_dependent(void (*kernel)(Params...), dim3 grid, int threads, cudaStream_t stream, Args... args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = dim3(unsigned(threads));
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, Params(args)...);
}

}  // namespace

}  // namespace gb200

using namespace gb200;

extern "C" {

int garnet_b200_gpt_oss_rms_norm(const float* d_x, const float* d_weight, float* d_y, int rows, int hidden, float epsilon, void* stream)
{
    if (!d_x || !d_weight || !d_y || rows <= 0 || hidden <= 0 || !(epsilon > 0.f))
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_rms_norm: bad argument");
    oss_rms_norm_kernel<<<rows, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_x, d_weight, d_y, hidden, epsilon);
    GB_CUDA(cudaGetLastError());
    return GARNET_B200_OK;
}

int garnet_b200_gpt_oss_rope(const garnet_b200_gpt_oss_options* o, const float* d_x, const long long* d_positions, float* d_y, int tokens,
                             void* stream)
{
    if (int rc = validate_oss(o, false)) return rc;
    if (!d_x || !d_positions || !d_y || tokens <= 0) return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_rope: bad argument");
    OssRope r{o->q_heads, o->kv_heads, o->head_dim, o->theta, o->factor, o->initial_context, o->beta_fast, o->beta_slow};
    // about two CTAs per SM at least: a decode batch shares the heads of a token over several CTAs
    const bool wide = o->head_dim % 8 == 0 && ((reinterpret_cast<uintptr_t>(d_x) | reinterpret_cast<uintptr_t>(d_y)) & 15) == 0;
    const int items = (o->q_heads + o->kv_heads) * o->head_dim / (wide ? 8 : 2), per_cta = tokens < 2 * kSmCount ? 1 : kRopeTokens,
              blocks = (tokens + per_cta - 1) / per_cta;
    const unsigned parts = unsigned(std::max(1, std::min((items + kRopeThreads - 1) / kRopeThreads, 2 * kSmCount / blocks)));
    // few tokens: little code, since a thread has one piece and fetches its instructions cold (4 tokens 7.4 -> 6.1 us)
    const auto kernel = !wide ? oss_rope_kernel<1, 1> : per_cta == 1 ? oss_rope_kernel<4, 1> : oss_rope_kernel<4, 3>;
    GB_CUDA(launch_dependent(kernel, dim3(unsigned(blocks), parts), kRopeThreads,
                             static_cast<cudaStream_t>(stream), d_x, d_positions, d_y, tokens, per_cta, r));
    return GARNET_B200_OK;
}

int garnet_b200_gpt_oss_attention_workspace(const garnet_b200_gpt_oss_options* o, int batch, int logical_pages, size_t* bytes)
{
    if (int rc = validate_oss(o, true)) return rc;
    if (!bytes || batch <= 0 || logical_pages <= 0) return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_attention_workspace: bad argument");
    *bytes = oss_workspace(*o, batch, logical_pages);
    return GARNET_B200_OK;
}

int garnet_b200_gpt_oss_attention(const garnet_b200_gpt_oss_options* o, const void* const* in, float* d_y, void* d_workspace,
                                  size_t workspace_bytes, int batch, int tokens, int logical_pages, int physical_pages, void* stream)
{
    if (int rc = validate_oss(o, true)) return rc;
    if (!in || !d_y || batch <= 0 || tokens <= 0 || logical_pages <= 0 || physical_pages <= 0)
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_attention: bad argument");
    for (int i = 0; i < 8; ++i)
        if (!in[i] && i != 4) return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_attention: operand %d is null", i);
    OssAttn p;
    p.qkv = static_cast<const float*>(in[0]);
    p.keys = static_cast<__nv_bfloat16*>(const_cast<void*>(in[1]));
    p.values = static_cast<__nv_bfloat16*>(const_cast<void*>(in[2]));
    p.table = static_cast<const int*>(in[3]);
    p.lengths = static_cast<const int*>(in[4]);
    p.starts = static_cast<const int*>(in[5]);
    p.active = static_cast<const int*>(in[6]);
    p.sinks = static_cast<const float*>(in[7]);
    p.out = d_y;
    p.batch = batch, p.tokens = tokens, p.logical_pages = logical_pages, p.physical_pages = physical_pages;
    p.q_heads = o->q_heads, p.kv_heads = o->kv_heads, p.head_dim = o->head_dim, p.layer = o->layer, p.page_size = o->page_size;
    p.window = o->window, p.prefill = o->prefill;
    cudaStream_t s = static_cast<cudaStream_t>(stream);
    const bool wide = o->head_dim % 8 == 0 && ((reinterpret_cast<uintptr_t>(in[0]) | reinterpret_cast<uintptr_t>(in[1]) |
                                                reinterpret_cast<uintptr_t>(in[2])) & 15) == 0;
    const size_t n = size_t(batch) * tokens * 2 * o->kv_heads * o->head_dim / (wide ? 8 : 1);
    GB_CUDA(launch_dependent(wide ? oss_write_kv_kernel<8> : oss_write_kv_kernel<1>, dim3(unsigned((n + 255) / 256)), 256, s, p));
    const int group = o->q_heads / o->kv_heads;
    const bool grouped = tokens == 1 && !o->prefill && o->head_dim == kOssDim && group <= 16 && in[4] &&
                         (reinterpret_cast<uintptr_t>(in[1]) & 15) == 0 && (reinterpret_cast<uintptr_t>(in[2]) & 15) == 0;
    if (grouped) {
        if (!d_workspace || workspace_bytes < oss_workspace(*o, batch, logical_pages) || (reinterpret_cast<uintptr_t>(d_workspace) & 255))
            return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_attention: the workspace is missing, too small or not 256-byte aligned");
        if (oss_decode_takes(p)) return oss_decode_launch(p, s);
    } else {
        if (!in[4] && !o->prefill) return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_attention: decode needs the lengths operand");
        if (o->head_dim > 256) return fail(GARNET_B200_NOT_SUPPORTED, "gpt_oss_attention: head_dim above 256");
    }
    if (oss_prefill_takes(p)) return oss_prefill_launch(p, s);
    const size_t tasks = size_t(batch) * tokens * o->q_heads;
    oss_attention_generic_kernel<<<unsigned((tasks * 32 + 255) / 256), 256, 0, s>>>(p);
    GB_CUDA(cudaGetLastError());
    return GARNET_B200_OK;
}

int garnet_b200_gpt_oss_vocab_top1(const float* d_logits, float* d_pairs, int rows, int width, int rank, void* stream)
{
    if (!d_logits || !d_pairs || rows <= 0 || width <= 0 || width > (1 << 23) || rank < 0)
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_vocab_top1: bad argument");
    oss_vocab_top1_kernel<<<rows, 256, 0, static_cast<cudaStream_t>(stream)>>>(d_logits, d_pairs, width, rank);
    GB_CUDA(cudaGetLastError());
    return GARNET_B200_OK;
}

int garnet_b200_gpt_oss_decode_gemv(const void* d_x, const void* d_weight, void* d_y, int rows, int columns, int weight_stride,
                                    int column_offset, int q_heads, int kv_heads, int head_dim, int rank, void* stream)
{
    if (!d_x || !d_weight || !d_y || rows <= 0 || columns <= 0 || columns % 32 != 0 || weight_stride < column_offset + columns ||
        column_offset < 0 ||
        (q_heads > 0 && (rank < 0 || rank > 1 || kv_heads <= 0 || head_dim <= 0 || q_heads % 2 || kv_heads % 2 ||
                         rows != (q_heads / 2 + kv_heads) * head_dim)))
        return fail(GARNET_B200_INVALID_VALUE, "gpt_oss_decode_gemv: bad argument");
    oss_gemv_kernel<<<unsigned((rows + 3) / 4), 128, 0, static_cast<cudaStream_t>(stream)>>>(
        static_cast<const __nv_bfloat16*>(d_x), static_cast<const __nv_bfloat16*>(d_weight), static_cast<__nv_bfloat16*>(d_y), rows,
        columns, weight_stride, column_offset, q_heads, kv_heads, head_dim, rank);
    GB_CUDA(cudaGetLastError());
    return GARNET_B200_OK;
}

}  // extern "C"
