// Small matrix products in 32-bit out of bfloat16 ones, for the recurrences that walk a sequence in chunks of tokens.
//
// A 32-bit number is held as the sum of three bfloat16 numbers (8 significant bits each, 24 in all: the split is
// exact but for the last half bit).  A product of an operand that is bfloat16 already with a split one takes three
// tensor-core products, one of two split operands six (those whose weight is above 2^-24 of the largest), each with 32-bit
// accumulation.  The tiles are those of mma.sync m16n8k16 (8.1 clocks each on a quarter of an SM): what a chunk multiplies is 16 to
// 32 rows of 64 or 128, with the state in registers between the products, too small and too dependent on one another for a
// 128-row tile in tensor memory.
#pragma once

#include "common.cuh"
#include "scan_wide.cuh"

namespace ff {

__device__ __forceinline__ uint32_t cm_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void cm_ldsm4(uint32_t r[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(cm_smem(p)) : "memory");
}
__device__ __forceinline__ void cm_ldsm4t(uint32_t r[4], const void* p) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(cm_smem(p)) : "memory");
}
__device__ __forceinline__ void cm_mma(float c[4], const uint32_t a[4], const uint32_t b[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}

// c += x and the columns of c times a pair, two columns an instruction: the warps of a walk have an instruction every second clock and
// no more, so what is not a product counts too
__device__ __forceinline__ void cm_add(float c[4], const float x[4]) {
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        const f32x2 r = f2_add(f2_pack(c[e], c[e + 1]), f2_pack(x[e], x[e + 1]));
        c[e] = f2_low(r);
        c[e + 1] = f2_high(r);
    }
}
__device__ __forceinline__ void cm_scale(float c[4], f32x2 by) {
#pragma unroll
    for (int e = 0; e < 4; e += 2) {
        const f32x2 r = f2_mul(f2_pack(c[e], c[e + 1]), by);
        c[e] = f2_low(r);
        c[e + 1] = f2_high(r);
    }
}

// c + small += A B with A held in NA parts and B in NB (1: bfloat16 as it is, 3: split).  The tensor core cuts its sums off
// instead of rounding them, always toward zero, and a chain of products on one accumulator adds that up.  So the products of
// the leading parts, which are 16 bits long and lose next to nothing among themselves, start from zero every time and are
// added to c with a rounded addition; all others, 2^-8 of them and less, are chained in `small`, which the caller adds to c
// at the end.
template <int NA, int NB>
__device__ __forceinline__ void cm_mma_parts(float c[4], float small[4], const uint32_t (&a)[NA][4], const uint32_t (&b)[NB][2]) {
    float t[4] = {0.f, 0.f, 0.f, 0.f};
    cm_mma(t, a[0], b[0]);
#pragma unroll
    for (int i = NA - 1; i >= 0; --i) {
#pragma unroll
        for (int j = NB - 1; j >= 0; --j)
            if (i + j == 1 || i + j == 2) cm_mma(small, a[i], b[j]);
    }
    cm_add(c, t);
}
// The same for two neighbouring tiles of eight columns, their right operand as ldmatrix gives it: r[part] = two registers of the
// first tile, two of the second.
template <int NA, int NB>
__device__ __forceinline__ void cm_mma_rows(float c[2][4], float small[2][4], const uint32_t (&a)[NA][4], const uint32_t (&r)[NB][4]) {
    uint32_t b0[NB][2], b1[NB][2];
#pragma unroll
    for (int p = 0; p < NB; ++p) { b0[p][0] = r[p][0]; b0[p][1] = r[p][1]; b1[p][0] = r[p][2]; b1[p][1] = r[p][3]; }
    cm_mma_parts<NA, NB>(c[0], small[0], a, b0);
    cm_mma_parts<NA, NB>(c[1], small[1], a, b1);
}

__device__ __forceinline__ uint32_t cm_pack(float lo, float hi) {      // (lo in the low half)
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ float cm_lo(uint32_t p) { return __uint_as_float(p << 16); }
__device__ __forceinline__ float cm_hi(uint32_t p) { return __uint_as_float(p & 0xffff0000u); }

// (x, y) as three packed pairs of bfloat16
__device__ __forceinline__ void cm_split3(float x, float y, uint32_t& p0, uint32_t& p1, uint32_t& p2) {
    const f32x2 minus = f2_pack(-1.f, -1.f);
    p0 = cm_pack(x, y);
    f32x2 rest = f2_fma(f2_pack(cm_lo(p0), cm_hi(p0)), minus, f2_pack(x, y));
    p1 = cm_pack(f2_low(rest), f2_high(rest));
    rest = f2_fma(f2_pack(cm_lo(p1), cm_hi(p1)), minus, rest);
    p2 = cm_pack(f2_low(rest), f2_high(rest));
}

// is one of the two bfloat16 numbers of `p` an infinity or not a number?
__device__ __forceinline__ bool cm_not_finite(uint32_t p) {
    return (p & 0x7f800000u) == 0x7f800000u || (p & 0x00007f80u) == 0x00007f80u;
}

// 16 bytes into shared memory, zeros where `in` is false (nothing is read then)
__device__ __forceinline__ void cm_copy16(void* dst, const void* src, bool in) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(cm_smem(dst)), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cm_copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cm_copy_wait() { asm volatile("cp.async.wait_group %0;" :: "n"(N) : "memory"); }

// barrier over `threads` threads of the block (whole warps); id 1 to 15
__device__ __forceinline__ void cm_barrier(int id, int threads) {
    asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(threads) : "memory");
}

}  // namespace ff
