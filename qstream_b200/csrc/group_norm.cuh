// A row's elements gated and normed in groups, in 16-byte pieces (the kernels behind the recurrences).
#pragma once

#include "common.cuh"

template <typename T>
__device__ __forceinline__ void store8(T* p, const float (&f)[8]) {
    if constexpr (sizeof(T) == 4) {
        reinterpret_cast<float4*>(p)[0] = make_float4(f[0], f[1], f[2], f[3]);
        reinterpret_cast<float4*>(p)[1] = make_float4(f[4], f[5], f[6], f[7]);
    } else {
        uint32_t u[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const __nv_bfloat162 r = __floats2bfloat162_rn(f[2 * j], f[2 * j + 1]);
            u[j] = *reinterpret_cast<const uint32_t*>(&r);
        }
        *reinterpret_cast<uint4*>(p) = make_uint4(u[0], u[1], u[2], u[3]);
    }
}

// out = v / sqrt(mean over a group of v^2 + eps) * w * act(gate), v = o;  SSD: v = (o + D x) silu(gate), no gate afterwards.
// A block per row; a thread holds NP pieces of eight neighbouring elements in registers from the loads to the store, all loads
// in flight together.  Groups are the whole row, or powers of two of at
// most 256 elements (the lanes of a group add up by shuffles); a group of 0: no norm.  Bound by memory: 4,096 rows of 2,048 from
// float32, one norm over the row, sigmoid gate, behind the scan: the whole mixer 623 -> 600 us (one element per thread and pass before).
template <typename TI, typename TG, typename TO, int NP, bool SSD>
__global__ void __launch_bounds__(256)
row_group_norm_kernel(TO* __restrict__ out, size_t ldo, const TI* __restrict__ o, size_t ldi, const void* __restrict__ w, int w_dtype,
                      const TG* __restrict__ gate, size_t ldg, int gate_act, int n, int group, float eps, int gate_span,
                      const TG* __restrict__ x, size_t ldx, const float* __restrict__ Dv, int dv) {
    __shared__ float scratch[33];
    grid_dep_launch();
    const size_t row = blockIdx.x;
    const int pieces = n >> 3;
    grid_dep_wait();
    constexpr int CI = sizeof(TI) == 4 ? QS_F32 : QS_BF16, CG = sizeof(TG) == 4 ? QS_F32 : QS_BF16;
    float v[NP][8], g[NP][8], wv[NP][8], xv[SSD ? NP : 1][8];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int p = threadIdx.x + i * blockDim.x;
#pragma unroll
        for (int j = 0; j < 8; ++j) v[i][j] = 0.f;
        if (p >= pieces) continue;
        load8_as_f32(o + row * ldi, CI, p * 8, v[i]);
        if (gate && gate_span == 1) load8_as_f32(gate + row * ldg, CG, p * 8, g[i]);
        else if (gate) g[i][0] = to_f32(gate[row * ldg + p * 8 / gate_span]);
        if (SSD) load8_as_f32(x + row * ldx, CG, p * 8, xv[i]);
        if (w) load8_as_f32(w, w_dtype, p * 8, wv[i]);
    }
    float total = 0.f, rstd[NP];
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int p = threadIdx.x + i * blockDim.x;
        float s = 0.f;
        if (SSD && p < pieces) {
            const float d = Dv[p * 8 / dv];
#pragma unroll
            for (int j = 0; j < 8; ++j) v[i][j] = fmaf(d, xv[i][j], v[i][j]) * silu_f32(g[i][j]);
        }
#pragma unroll
        for (int j = 0; j < 8; ++j) s = fmaf(v[i][j], v[i][j], s);
        if (group > 0 && group < n) {
            for (int off = group >> 4; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
            rstd[i] = 1.0f / sqrtf(s / (float)group + eps);
        }
        total += s;
    }
    if (group == n) {
        total = 1.0f / sqrtf(block_sum(total, scratch) / (float)n + eps);
#pragma unroll
        for (int i = 0; i < NP; ++i) rstd[i] = total;
    }
#pragma unroll
    for (int i = 0; i < NP; ++i) {
        const int p = threadIdx.x + i * blockDim.x;
        if (p >= pieces) continue;
        const float one = !SSD && gate && gate_span > 1 ? apply_activation(g[i][0], gate_act) : 1.0f;
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            float y = v[i][j];
            if (group > 0) y *= rstd[i];
            if (w) y *= wv[i][j];
            if (!SSD && gate) y *= gate_span > 1 ? one : apply_activation(g[i][j], gate_act);
            v[i][j] = y;
        }
        store8(out + row * ldo + p * 8, v[i]);
    }
}

// Whether the kernel above takes a row of n elements in groups of `group`, spans of `gate_span`; rows of fewer than `fewest` elements are
// the general kernels'.
inline bool row_group_norm_takes(int n, int group, int gate_span, int fewest) {
    const bool pow2 = group >= 8 && group <= 256 && (group & (group - 1)) == 0;
    return n % 8 == 0 && n >= fewest && n <= 8 * 256 * 4 && (group == 0 || group == n || pow2) && (gate_span == 1 || gate_span % 8 == 0);
}
template <typename T>
inline bool in_pieces(const T* p, long long ld) { return !p || (((uintptr_t)p % 16) == 0 && ld % 8 == 0); }

template <typename TI, typename TG, typename TO, bool SSD>
cudaError_t launch_row_group_norm(TO* out, size_t ldo, const TI* o, size_t ldi, const void* w, int w_dtype, const TG* gate, size_t ldg, int gate_act,
                                  int rows, int n, int group, float eps, int gate_span, const TG* x, size_t ldx, const float* Dv, int dv,
                                  cudaStream_t stream) {
    const int pieces = n / 8, np = pieces <= 256 ? 1 : (pieces <= 512 ? 2 : 4), threads = ((pieces + np - 1) / np + 31) / 32 * 32;
#define QS_GO(NP) return qs_launch_dependent(row_group_norm_kernel<TI, TG, TO, NP, SSD>, dim3(rows), dim3(threads), 0, stream, out, ldo, o, ldi, w, w_dtype, \
        gate, ldg, gate_act, n, group, eps, gate_span, x, ldx, Dv, dv)
    if (np == 1) QS_GO(1);
    if (np == 2) QS_GO(2);
    QS_GO(4);
#undef QS_GO
}
