// What the 32-bit products share: the end of an output element, and the sum of a product's parts along K.
#pragma once

#include "common.cuh"

namespace {

template <typename TA, typename TC>
__device__ __forceinline__ void finish(TC* __restrict__ C, float v, int gm, int gn, const void* __restrict__ bias, int bias_dtype, int act,
                                       const TA* __restrict__ res1, const TA* __restrict__ res2, size_t ldc, size_t ldr) {
    if (bias) v += load_as_f32(bias, bias_dtype, gn);
    v = apply_activation(v, act);
    if (res1) v += to_f32(res1[(size_t)gm * ldr + gn]);
    if (res2) v += to_f32(res2[(size_t)gm * ldr + gn]);
    C[(size_t)gm * ldc + gn] = from_f32<TC>(v);
}

// C = act(sum of the runs' sums, in order, + bias) + residuals.
template <typename TA, typename TC>
__global__ void __launch_bounds__(256)
linear_join_kernel(TC* __restrict__ C, const float* __restrict__ partial, int runs, const void* __restrict__ bias, int bias_dtype, int act,
                   const TA* __restrict__ res1, const TA* __restrict__ res2, int M, int N, size_t ldc, size_t ldr) {
    const size_t mn = (size_t)M * N;
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < mn; e += (size_t)gridDim.x * blockDim.x) {
        float total = 0.f;
        int r = 0;
        for (; r + 8 <= runs; r += 8) {                     // eight loads in flight
            float v[8];
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = partial[(r + i) * mn + e];
#pragma unroll
            for (int i = 0; i < 8; ++i) total += v[i];
        }
        for (; r < runs; ++r) total += partial[r * mn + e];
        finish(C, total, (int)(e / N), (int)(e % N), bias, bias_dtype, act, res1, res2, ldc, ldr);
    }
}

}  // namespace
