// 32-bit numbers as sums of three bfloat16 terms, h + m + l, each the rounded rest of the one before: all 24 bits of a number whose rest does not
// underflow.  Products of 32-bit numbers are then exact products of terms (hh, hm, mh, mm, hl, lh; what is left out is below 2^-26
// of the product), which the tensor cores add up.  The unit cuts off where it adds; so it sums a few products from zero, small terms
// first, and those sums are added outside with rounded 32-bit additions.  A number that is not finite, or rounds to infinity as
// bfloat16, has no such terms: its last one is NaN, and with it every sum that it takes part in.  Below 2^-109 the last term is cut, as a bfloat16 ends
// at 2^-133.
#pragma once

#include "common.cuh"

namespace {

__device__ __forceinline__ uint32_t pack_bf16(float2 v) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(v.y), "f"(v.x));
    return r;
}
__device__ __forceinline__ f32x2 widen(uint32_t p) { return pack2(__uint_as_float(p << 16), __uint_as_float(p & 0xffff0000u)); }

// Two numbers' terms, each pair in a word.
__device__ __forceinline__ void terms_of(f32x2 v, uint32_t& h, uint32_t& m, uint32_t& l) {
    const f32x2 minus = pack2(-1.f, -1.f);
    h = pack_bf16(unpack2(v));
    const f32x2 rest = fma2(widen(h), minus, v);
    m = pack_bf16(unpack2(rest));
    l = pack_bf16(unpack2(fma2(widen(m), minus, rest)));
}

// Whether a sum of products of terms can be taken as it is: a number, and zero or so large that the operands which decide it were held whole (16,384
// products of numbers below 2^-109 and below 2^31 stay under the limit).  Else it is taken again from the 32-bit numbers, by multiply-adds.
// `beyond`: up to HELD for all of these but zero, above it for the rest; the largest over many sums is two instructions each where three comparisons
// each cost the scans 3 to 4 %.
constexpr uint32_t HELD = 0xbffffffeu;                  // the largest number less 2^-64, bits without the sign
__device__ __forceinline__ uint32_t beyond(float sum) { return (__float_as_uint(sum) << 1) - 0x3f000000u; }
__device__ __forceinline__ bool held(float sum) { return beyond(sum) <= HELD || sum == 0.f; }

// ---- tiles of terms in shared memory as operands of mma.sync

__device__ __forceinline__ void load_matrices(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void load_matrices_turned(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}

// Where a lane points for the four 8 x 8 matrices of a piece of 16 x 16 elements that begins at (r, c) of a tile [rows][pitch] of bfloat16:
// as an A operand stored [m][k] and as two B operands stored [k][n] (turned), the matrices go down the rows first;
__device__ __forceinline__ int rows_first(int r, int c, int pitch, int lane) { return ((r + (lane & 15)) * pitch + c + (lane >> 4) * 8) * 2; }
// as an A operand stored [k][m] (turned) and as two B operands stored [n][k], across the columns first.
__device__ __forceinline__ int columns_first(int r, int c, int pitch, int lane) { return ((r + (lane & 7) + (lane >> 4) * 8) * pitch + c + (lane >> 3 & 1) * 8) * 2; }

__device__ __forceinline__ void mma_onto(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

// sum += A B over 16 products, A and B in PA and PB terms: the unit's part from zero, small products first, then one rounded addition.  `n`: which
// of the two B operands of `b`.
template <int PA, int PB>
__device__ __forceinline__ void add_product(float (&sum)[4], const uint32_t (&a)[PA][4], const uint32_t (&b)[PB][4], int n) {
    float d[4];
    bool first = true;
#pragma unroll
    for (int order = PA + PB - 2; order >= 0; --order)
#pragma unroll
        for (int x = 0; x < PA; ++x) {
            const int y = order - x;
            if (order > 2 || y < 0 || y >= PB) continue;
            if (first) mma_bf16_16x8x16(d, a[x][0], a[x][1], a[x][2], a[x][3], b[y][2 * n], b[y][2 * n + 1]);
            else mma_onto(d, a[x], b[y][2 * n], b[y][2 * n + 1]);
            first = false;
        }
#pragma unroll
    for (int i = 0; i < 4; ++i) sum[i] += d[i];
}

}  // namespace
