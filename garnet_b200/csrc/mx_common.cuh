// Helpers shared by the block-scaled (tcgen05.mma kind::mxf8f6f4) MoE kernels.
#pragma once
#include "tc_common.cuh"

namespace gb200 {

constexpr int kMxSlab = 128;         // K elements per pipeline stage (4 MMAs of K = 32 per piece)
constexpr int kMxAtom = 512;         // bytes of one scale atom: 128 rows x 4 blocks
constexpr int kMxMaxExperts = 1024;
// Rows that one TMA of a row tile's piece brings, by how many the tile holds (moe_mxr.cu says what hangs on it).  The second
// pieces' scales of a small tile follow the first ones' in its scale atoms, `box` rows on.
constexpr int kMxBoxSmall = 32, kMxBoxMid = 56, kMxBoxFull = 128;
__host__ __device__ constexpr int mx_tile_box(int rows) { return rows <= kMxBoxSmall ? kMxBoxSmall : rows <= kMxBoxMid ? kMxBoxMid : kMxBoxFull; }

#if defined(__CUDACC__)

// K-major operand without swizzle: 8-row core matrices of 128 contiguous bytes, 128 bytes apart (the source format of the
// scale-atom copies):
constexpr uint32_t kMxPlainHi = (128u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t mx_plain_lo(uint32_t smem_addr) { return (smem_addr & 0x3FFFFu) >> 4; }

// 32 rows x 16 bytes of shared memory -> 4 columns of tensor memory, replicated to
// the four 32-lane quarters.
__device__ __forceinline__ void tmem_cp_32x128b_warpx4(uint32_t taddr, uint32_t src_lo)
{
    asm volatile(
        "{\n\t.reg .b64 d;\n\t"
        "mov.b64 d, {%1, %2};\n\t"
        "tcgen05.cp.cta_group::1.32x128b.warpx4 [%0], d;\n\t}" ::"r"(taddr), "r"(src_lo), "n"(kMxPlainHi)
        : "memory");
}

// Instruction descriptor of kind::mxf8f6f4, both operands K-major, e8m0 scales; operand
// formats: 0 = e4m3, 5 = e2m1; `sf` selects which of the four blocks of the scale atoms
// this MMA uses.
constexpr uint32_t kMxFmtE4M3 = 0, kMxFmtE2M1 = 5;
__host__ __device__ constexpr uint32_t mx_idesc_fmt(uint32_t a_fmt, uint32_t b_fmt, int m, int n, uint32_t sf)
{
    return (sf << 4) | (a_fmt << 7) | (b_fmt << 10) | (uint32_t(n >> 3) << 17) | (1u << 23) | (uint32_t(m >> 4) << 24) | (sf << 29);
}

__device__ __forceinline__ void umma_mx(uint32_t d_tmem, uint32_t a_lo, uint32_t b_lo, uint32_t idesc, uint32_t sfa,
                                        uint32_t sfb, bool accumulate)
{
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 a, b;\n\t"
        "mov.b64 a, {%1, %7};\n\tmov.b64 b, {%2, %7};\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf8f6f4.block_scale [%0], a, b, %3, [%5], [%6], p;\n\t}" ::"r"(d_tmem),
        "r"(a_lo), "r"(b_lo), "r"(idesc), "r"(uint32_t(accumulate)), "r"(sfa), "r"(sfb), "n"(kDescHiSw128)
        : "memory");
}

__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, uint32_t (&r)[8])
{
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

#endif  // __CUDACC__

}  // namespace gb200
