// Chunks of 64 tokens: loads, staged tiles and the sums over pairs of tokens with a decay per channel, on the CUDA cores.
#pragma once

#include "common.cuh"

namespace {

constexpr int CT = 64;                                  // tokens of a chunk
constexpr int PP = CT + 4;                              // pitch of a chunk's weights P[j][t]

// Where channel c's column of a staged [channels][64 tokens] tile lies: tokens in groups of four, permuted by the channel's
// group of four, so that a warp that writes 8 x 4 channels of four tokens meets every bank once.
__device__ __forceinline__ int at_ct(int c, int t) { return c * CT + (t ^ (((c >> 2) & 7) << 2)); }

// Four neighbouring elements of a row, zeros behind its end: fetched in one step and turned into 32-bit numbers in another, so that
// many fetches are under way before the first is waited for.
template <typename TI> struct Raw4;
template <> struct Raw4<float> {
    float4 x;
    __device__ __forceinline__ void get(const float* p) { x = *reinterpret_cast<const float4*>(p); }
    __device__ __forceinline__ void zero() { x = make_float4(0.f, 0.f, 0.f, 0.f); }
    __device__ __forceinline__ float4 value() const { return x; }
};
template <> struct Raw4<__nv_bfloat16> {
    uint2 x;
    __device__ __forceinline__ void get(const __nv_bfloat16* p) { x = *reinterpret_cast<const uint2*>(p); }
    __device__ __forceinline__ void zero() { x = make_uint2(0u, 0u); }
    __device__ __forceinline__ float4 value() const {
        return make_float4(__uint_as_float(x.x << 16), __uint_as_float(x.x & 0xffff0000u), __uint_as_float(x.y << 16), __uint_as_float(x.y & 0xffff0000u));
    }
};
template <typename TI>
__device__ __forceinline__ void get_four(Raw4<TI>& r, const TI* __restrict__ row, int i, int n, bool have, int vec) {
    if (!have || i >= n) { r.zero(); return; }
    if (vec) { r.get(row + i); return; }
    TI f[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) f[j] = i + j < n ? row[i + j] : from_f32<TI>(0.f);
    if constexpr (sizeof(TI) == 4) r.x = make_float4(f[0], f[1], f[2], f[3]);
    else {
        const __nv_bfloat162 a = __halves2bfloat162(f[0], f[1]), b = __halves2bfloat162(f[2], f[3]);
        r.x = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
    }
}
__device__ __forceinline__ void copy16(float* dst, const float* src, bool have) {       // asynchronous; zeros where there is nothing
    if (have) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
    else *reinterpret_cast<float4*>(dst) = make_float4(0.f, 0.f, 0.f, 0.f);
}
__device__ __forceinline__ void copies_done() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Sums over pairs of tokens in different blocks of 16: [16 t][16 I j] of block I with rows of 16 I + 1 (they are read along t)
constexpr int CROSS = 16 * (17 + 33 + 49);
// acc[x][pair of t] += sum over N channels from c0 on of X[i][t] k[i][j]: block I's tokens t = 4 (lane / 8) .. + 3 against the earlier
// blocks' tokens j = 16 m + 2 (lane % 8) + {0, 1}, x = 2 m + {0, 1}
template <int I, int N, int (*AT)(int, int)>
__device__ __forceinline__ void cross_product(f32x2 (&acc)[2 * I][2], const float* __restrict__ X, const float* __restrict__ sk, int c0, int lane) {
#pragma unroll 4
    for (int i = c0; i < c0 + N; ++i) {
        const ulonglong2 a = *reinterpret_cast<const ulonglong2*>(X + AT(i, I * 16 + (lane >> 3) * 4));
#pragma unroll
        for (int m = 0; m < I; ++m) {
            const float2 b = *reinterpret_cast<const float2*>(sk + AT(i, m * 16 + (lane & 7) * 2));
            const f32x2 b0 = pack2(b.x, b.x), b1 = pack2(b.y, b.y);
            acc[2 * m][0] = fma2(a.x, b0, acc[2 * m][0]);
            acc[2 * m][1] = fma2(a.y, b0, acc[2 * m][1]);
            acc[2 * m + 1][0] = fma2(a.x, b1, acc[2 * m + 1][0]);
            acc[2 * m + 1][1] = fma2(a.y, b1, acc[2 * m + 1][1]);
        }
    }
}
__device__ __forceinline__ int cross_at(int I) { return 16 * (8 * I * (I - 1) + I - 1); }      // where block I's sums begin
template <int I>
__device__ __forceinline__ void cross_store(float* __restrict__ dst, const f32x2 (&acc)[2 * I][2], int lane) {
    dst += cross_at(I);
#pragma unroll
    for (int x = 0; x < 2 * I; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const float2 v = unpack2(acc[x][y]);
            float* at = dst + ((lane >> 3) * 4 + 2 * y) * (16 * I + 1) + (x >> 1) * 16 + (lane & 7) * 2 + (x & 1);
            at[0] = v.x;
            at[16 * I + 1] = v.y;
        }
}
// four tokens of a channel times a decay
__device__ __forceinline__ void scale_four(float* at, float d) {
    float4 v = *reinterpret_cast<float4*>(at);
    v.x *= d; v.y *= d; v.z *= d; v.w *= d;
    *reinterpret_cast<float4*>(at) = v;
}

}  // namespace
