// Float32 matrix products on the tensor cores: every operand in three bfloat16 parts whose sum is the float32 number
// (x = hi + mid + lo, each part the rounding of what the parts before leave: 3 x 8 bits), six of the nine part products
// (hi hi, hi mid, mid hi, mid mid, hi lo, lo hi; what is left out is 2^-23 of the product at most, 2^-27 rms).  The method is that of Henry, Tang and Heinecke, "Leveraging the bfloat16
// artificial intelligence datatype for higher-precision computations" (2019).  The third part of a number below 2^-109 falls under the smallest bfloat16 number,
// 2^-133: such a number is kept to 2^-134, which shows only in sums that are as small.
//
// The tensor cores add with truncation at 2^-25 of the largest term, and truncate every accumulation again, so a long chain of
// accumulations drifts towards zero.  Therefore hi hi is taken from zero for every 16 k and added up in registers with
// rounding (a sum of 16 products of 8-bit numbers from zero: 0.34 units of 2^-24 rms, one of 16 fused multiply-adds 0.30), and
// the five others, 2^-8 of it at most, have an accumulator of their own.
//
// Rate: an SM issues 1,020 bfloat16 multiply-adds a cycle through mma.sync (measured), 170 of these products; its FMA units 128 at best and
// 50 to 70 in the loops this replaces.  tcgen05.mma multiplies four times as fast, and sums of 64 k in tensor memory are close enough (gemm_split.cu);
// here it would take the state's parts through shared memory for every chunk, which is not built.
#pragma once
#include <stdint.h>

struct SplitA { uint32_t hi[4], mid[4], lo[4]; };               // an operand of 16 rows x 16 k (mma.m16n8k16 A)

__device__ __forceinline__ uint32_t split_pack(float even, float odd) {
    uint32_t out;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(out) : "f"(odd), "f"(even));
    return out;
}
// the numbers of k and k + 1 of a row
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = split_pack(a, b);
    a -= __uint_as_float(hi << 16);
    b -= __uint_as_float(hi & 0xffff0000u);
    mid = split_pack(a, b);
    a -= __uint_as_float(mid << 16);
    b -= __uint_as_float(mid & 0xffff0000u);
    lo = split_pack(a, b);
}

__device__ __forceinline__ void split_mma(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void split_mma_zero(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1), "f"(0.0f));
}
// from zero, then added with rounding
__device__ __forceinline__ void split_mma_add(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    float t[4];
    split_mma_zero(t, a, b0, b1);
    d[0] += t[0]; d[1] += t[1]; d[2] += t[2]; d[3] += t[3];
}

// The other operand lies in memory as the lanes take it: for 16 k and two tiles of 8 columns, three pieces (hi, mid, lo) of 32 lanes x 16
// bytes: {k and k + 1, k + 8 and k + 9} of the first tile's column, then of the second's (k = 2 (lane % 4), column = lane / 4).
constexpr int SPLIT_BLOCK_BYTES = 3 * 512;

// main, rest [2 BLOCKS tiles] += A (16 x 16) * BLOCKS neighbouring blocks B (16 x 16 each, at `block`); FIRST: = instead of +=.  Products that
// add to the same numbers are 2 BLOCKS instructions apart: one alone takes 20 cycles, a new one may start every 8.
template <int BLOCKS, bool FIRST>
__device__ __forceinline__ void split_products(float (*main)[4], float (*rest)[4], const SplitA& a, const uint4* block, int lane) {
    uint4 hi[BLOCKS], mid[BLOCKS], lo[BLOCKS];
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) { hi[k] = block[k * 96 + lane]; lo[k] = block[k * 96 + 64 + lane]; mid[k] = block[k * 96 + 32 + lane]; }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) {
        if (FIRST) { split_mma_zero(rest[2 * k], a.lo, hi[k].x, hi[k].y); split_mma_zero(rest[2 * k + 1], a.lo, hi[k].z, hi[k].w); }
        else { split_mma(rest[2 * k], a.lo, hi[k].x, hi[k].y); split_mma(rest[2 * k + 1], a.lo, hi[k].z, hi[k].w); }
    }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) {
        if (FIRST) { split_mma_zero(main[2 * k], a.hi, hi[k].x, hi[k].y); split_mma_zero(main[2 * k + 1], a.hi, hi[k].z, hi[k].w); }
        else { split_mma_add(main[2 * k], a.hi, hi[k].x, hi[k].y); split_mma_add(main[2 * k + 1], a.hi, hi[k].z, hi[k].w); }
    }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) { split_mma(rest[2 * k], a.hi, lo[k].x, lo[k].y); split_mma(rest[2 * k + 1], a.hi, lo[k].z, lo[k].w); }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) { split_mma(rest[2 * k], a.mid, mid[k].x, mid[k].y); split_mma(rest[2 * k + 1], a.mid, mid[k].z, mid[k].w); }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) { split_mma(rest[2 * k], a.mid, hi[k].x, hi[k].y); split_mma(rest[2 * k + 1], a.mid, hi[k].z, hi[k].w); }
#pragma unroll
    for (int k = 0; k < BLOCKS; ++k) { split_mma(rest[2 * k], a.hi, mid[k].x, mid[k].y); split_mma(rest[2 * k + 1], a.hi, mid[k].z, mid[k].w); }
}

// the other operand's parts as a warp's lanes hold them, in memory: three pieces (hi, mid, lo) of 32 lanes x 16 bytes
__device__ __forceinline__ void split_store(uint4* block, int lane, const SplitA& a) {
    block[lane] = make_uint4(a.hi[0], a.hi[1], a.hi[2], a.hi[3]);
    block[32 + lane] = make_uint4(a.mid[0], a.mid[1], a.mid[2], a.mid[3]);
    block[64 + lane] = make_uint4(a.lo[0], a.lo[1], a.lo[2], a.lo[3]);
}
__device__ __forceinline__ void split_load(SplitA& a, const uint4* block, int lane) {
    const uint4 hi = block[lane], mid = block[32 + lane], lo = block[64 + lane];
    a.hi[0] = hi.x; a.hi[1] = hi.y; a.hi[2] = hi.z; a.hi[3] = hi.w;
    a.mid[0] = mid.x; a.mid[1] = mid.y; a.mid[2] = mid.z; a.mid[3] = mid.w;
    a.lo[0] = lo.x; a.lo[1] = lo.y; a.lo[2] = lo.z; a.lo[3] = lo.w;
}

// writes such a block: v[tile][4] = the numbers of k, k + 1, k + 8, k + 9 of this lane's column of the tile
__device__ __forceinline__ void split_store(uint4* block, int lane, const float (&v)[2][4]) {
    uint4 hi, mid, lo;
    split_pair(v[0][0], v[0][1], hi.x, mid.x, lo.x);
    split_pair(v[0][2], v[0][3], hi.y, mid.y, lo.y);
    split_pair(v[1][0], v[1][1], hi.z, mid.z, lo.z);
    split_pair(v[1][2], v[1][3], hi.w, mid.w, lo.w);
    block[lane] = hi;
    block[32 + lane] = mid;
    block[64 + lane] = lo;
}
