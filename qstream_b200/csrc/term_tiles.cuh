// Tiles of 64 x 64 numbers as terms (terms.cuh) in shared memory, as tcgen05 operands: what the kernels over a prompt's chunks share.
#pragma once

#include "scan_tiles.cuh"
#include "sm100.cuh"
#include "terms.cuh"

using namespace sm100;

namespace {

// ---- tiles of terms in shared memory as tcgen05 operands: 64 elements to a row of 128 bytes, swizzled by 128 bytes.  A tile of
// 64 rows is 8 KB; wider ones are several of them.  The same tile serves with its rows on the sum's side or on the other.
constexpr int TILE = CT * 128;                          // bytes
constexpr uint32_t A_TURNED = 1u << 15, B_TURNED = 1u << 16;       // instruction descriptor: rows on the sum's side

__device__ __forceinline__ uint32_t place_in_tile(int r, int c) { return (uint32_t)(r * 128 + ((((c >> 3) ^ r) & 7) << 4) + (c & 7) * 2); }

// Four neighbouring numbers as terms at dst, dst + term ...  P = 1: they come as bfloat16.
template <int P>
__device__ __forceinline__ void put_terms(uint32_t dst, uint32_t term, float4 f) {
    uint32_t a[3], b[3];
    terms_of(pack2(f.x, f.y), a[0], a[1], a[2]);
    terms_of(pack2(f.z, f.w), b[0], b[1], b[2]);
#pragma unroll
    for (int i = 0; i < P; ++i) asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + i * term), "r"(a[i]), "r"(b[i]) : "memory");
}
// Eight neighbouring numbers as terms.
__device__ __forceinline__ void put_eight(uint32_t dst, uint32_t term, const float (&f)[8]) {
    uint32_t t[3][4];
#pragma unroll
    for (int j = 0; j < 4; ++j) terms_of(pack2(f[2 * j], f[2 * j + 1]), t[0][j], t[1][j], t[2][j]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(dst + i * term), "r"(t[i][0]), "r"(t[i][1]), "r"(t[i][2]), "r"(t[i][3]) : "memory");
}

// D (+)= A B over 64 products, A in PA terms that lie `a_term` apart, B in PB: small products first, from zero.  TURNED operands: rows on the
// sum's side, 64 elements of the other side per tile; else the sum along the rows.
template <int PA, int PB, bool A_T, bool B_T>
__device__ __forceinline__ void multiply_tiles(uint32_t d, uint32_t a, uint32_t a_term, uint32_t b, uint32_t b_term, int N) {
    const uint32_t idesc = idesc_bf16_f32(128, N) | (A_T ? A_TURNED : 0u) | (B_T ? B_TURNED : 0u);
    bool first = true;
#pragma unroll
    for (int order = 2; order >= 0; --order)
#pragma unroll
        for (int x = 0; x < PA; ++x) {
            const int y = order - x;
            if (y < 0 || y >= PB) continue;
            const uint32_t at = a + x * a_term, bt = b + y * b_term;
            const uint64_t da = A_T ? smem_desc_sw128_mn(at, TILE, 1024) : smem_desc_sw128(at), db = B_T ? smem_desc_sw128_mn(bt, TILE, 1024) : smem_desc_sw128(bt);
#pragma unroll
            for (int k = 0; k < 4; ++k) {               // 16 of the sum's elements: 32 bytes of a row, or two groups of eight rows
                mma_bf16(d, da + (A_T ? 128 : 2) * k, db + (B_T ? 128 : 2) * k, idesc, !first);
                first = false;
            }
        }
}

__device__ __forceinline__ bool wait_done(uint64_t* bar, uint32_t parity, int32_t* status) {
    if (__all_sync(0xffffffffu, mbar_wait(bar, parity))) return true;
    atomicExch(status, 171);
    return false;
}
// sum[0 .. N) += the thread's lane, columns from `taddr` on
template <int N>
__device__ __forceinline__ void take_sums(float (&sum)[N], uint32_t taddr, bool first) {
#pragma unroll
    for (int c = 0; c < N; c += 16) {
        uint32_t raw[16];
        tmem_load_32x16(taddr + c, raw);
        tmem_load_wait();
#pragma unroll
        for (int j = 0; j < 16; ++j) sum[c + j] = first ? __uint_as_float(raw[j]) : sum[c + j] + __uint_as_float(raw[j]);
    }
}

}  // namespace
