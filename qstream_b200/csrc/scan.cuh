// Shared by the walk in order (recurrent.cu) and the chunks of long prompts (scan_chunks.cu).
#pragma once

#include "common.cuh"

// One way for both signs: lanes of a warp that differ would take both.
__device__ __forceinline__ float log_sigmoid_f32(float z) { return fminf(z, 0.f) - log1pf(expf(-fabsf(z))); }

int qs_scan_chunks(int mode, int outputs, float* o, long long ldo, const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                   int dtype, const float* dlog, long long ldd, const float* head_decay, const void* bonus, int bonus_dtype, int H, int dk, int dv,
                   const int32_t* chunk_start, int n_chunks, int T_rows, float* chunk_state, float* chunk_decay, const float* ga, const float* gb,
                   long long ldg, float q_scale, int qk_group, float decay_scale, float* chunk_factors, int32_t* status, cudaStream_t stream);
