// Routed experts: the router's choice, and the two ways the chosen experts run.
//
//   moe_route     per token: scores s = sigmoid(z); choice scores s + correction; experts in equal groups of
//                 neighbours, a group's score the sum of its two largest choice scores, only the best `keep` groups
//                 stay (the others count as minus infinity); the `top` largest choice scores win (equal scores: the
//                 lower index); weights s * scale of the winners, not renormalised; optionally sigmoid of one more
//                 logit per token (the gate of a shared expert).  `score_kind` 1: s = softmax(z) over all experts
//                 instead of the sigmoid; `group_kind` 1: a group's score is its largest choice score; `renorm_eps` >= 0:
//                 the winners' scores are divided by their sum + renorm_eps
//   few tokens    moe_expert_up / moe_expert_down: every (token, chosen expert) pair reads its expert's matrices
//                 through the routing table on the device, so a step can be captured and replayed
//   many tokens   moe_sort orders the pairs by expert; the caller runs one matrix product per expert over its rows
//                 and moe_combine adds each token's weighted results
//   identity      a router may have more outputs than there are experts with matrices: the outputs behind the last expert
//                 return the token's own input, times the weight
//
// Router arithmetic, weights and all sums are 32-bit; a token's sum runs over its experts in the order of choice.
#include "common.cuh"

namespace {

constexpr int MAX_EXPERTS = 1024;

// One warp per token.  Lanes compute the scores; lane 0 selects.
__global__ void moe_route_kernel(int32_t* __restrict__ idx, float* __restrict__ wts, float* __restrict__ shared_gate,
                                 const float* __restrict__ z, size_t ldz, const void* __restrict__ corr, int corr_dtype,
                                 int T, int E, int top, int groups, int keep, float scale, int gate_col, int score_kind,
                                 int group_kind, float renorm_eps) {
    extern __shared__ float sm[];                       // per warp: s [E], choice [E], group score [groups]
    grid_dep_launch();
    grid_dep_wait();
    const int warps = blockDim.x >> 5, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * warps + warp;
    if (t >= T) return;
    float* s = sm + (size_t)warp * (2 * E + groups);
    float* choice = s + E;
    float* gscore = choice + E;
    const float* zr = z + (size_t)t * ldz;
    float z_max = -INFINITY, inv_sum = 1.0f;
    if (score_kind == 1) {                              // softmax over all experts: the largest logit, then the sum
        for (int e = lane; e < E; e += 32) z_max = fmaxf(z_max, zr[e]);
        for (int off = 16; off > 0; off >>= 1) z_max = fmaxf(z_max, __shfl_xor_sync(0xffffffffu, z_max, off));
        float sum = 0.f;
        for (int e = lane; e < E; e += 32) sum += expf(zr[e] - z_max);
        inv_sum = 1.0f / warp_sum(sum);
    }
    for (int e = lane; e < E; e += 32) {
        s[e] = score_kind == 1 ? expf(zr[e] - z_max) * inv_sum : sigmoid_f32(zr[e]);
        choice[e] = s[e] + (corr ? load_as_f32(corr, corr_dtype, e) : 0.f);
    }
    if (shared_gate && lane == 0 && gate_col >= 0) shared_gate[t] = sigmoid_f32(zr[gate_col]);
    __syncwarp();
    const int per = E / groups;
    if (keep < groups) {
        for (int g = lane; g < groups; g += 32) {
            float a = -INFINITY, b = -INFINITY;          // the two largest
            for (int e = g * per; e < (g + 1) * per; ++e) {
                const float c = choice[e];
                if (c > a) { b = a; a = c; } else if (c > b) b = c;
            }
            gscore[g] = (per > 1 && group_kind == 0) ? a + b : a;
        }
        __syncwarp();
        if (lane == 0) {
            // keep the best `keep` groups: drop the others' experts
            for (int n = 0; n < groups - keep; ++n) {
                int worst = -1;
                for (int g = 0; g < groups; ++g)            // the lowest score; among equals the highest index goes
                    if (gscore[g] != INFINITY && (worst < 0 || gscore[g] <= gscore[worst])) worst = g;
                gscore[worst] = INFINITY;                   // marks a dropped group
                for (int e = worst * per; e < (worst + 1) * per; ++e) choice[e] = -INFINITY;
            }
        }
        __syncwarp();
    }
    // The `top` largest, one after the other: lanes look over every 32nd expert, the warp takes the largest of theirs (equal scores: the
    // lower index).  NaN is larger than nothing and, as the first live expert, beaten by nothing, as in a walk in order.
    for (int j = 0; j < top; ++j) {
        float v = -INFINITY;
        int best = MAX_EXPERTS, first = MAX_EXPERTS;
        for (int e = lane; e < E; e += 32) {
            const float c = choice[e];
            if (c == -INFINITY) continue;
            if (first == MAX_EXPERTS) first = e;
            if (c > v) { v = c; best = e; }
        }
#pragma unroll
        for (int off = 16; off > 0; off >>= 1) {
            const float ov = __shfl_xor_sync(0xffffffffu, v, off);
            const int oe = __shfl_xor_sync(0xffffffffu, best, off);
            if (ov > v || (ov == v && oe < best)) { v = ov; best = oe; }
            first = min(first, __shfl_xor_sync(0xffffffffu, first, off));
        }
        if (first < MAX_EXPERTS && (best == MAX_EXPERTS || choice[first] != choice[first])) best = first;
        if (best == MAX_EXPERTS) best = 0;              // fewer live experts than `top`: cannot happen with a sound config
        __syncwarp();
        if (lane == 0) {
            idx[(size_t)t * top + j] = best;
            wts[(size_t)t * top + j] = s[best] * scale;
            choice[best] = -INFINITY;
        }
        __syncwarp();
    }
    if (lane == 0) {
        if (renorm_eps >= 0.f) {                            // the chosen scores made to sum to one, in the order of choice
            float sum = 0.f;
            for (int j = 0; j < top; ++j) sum += s[idx[(size_t)t * top + j]];
            const float inv = scale / (sum + renorm_eps);
            for (int j = 0; j < top; ++j) wts[(size_t)t * top + j] = s[idx[(size_t)t * top + j]] * inv;
        }
    }
}

// sum_k w[k] * x[k] over a warp: lanes take pieces of eight elements (16-byte loads of bfloat16, two of float32)
// where `vec` says that K is a multiple of 8 and the row is aligned, else single elements.
template <typename T>
__device__ __forceinline__ float warp_dot(const T* __restrict__ w, const float* __restrict__ x, int K, int lane, bool vec) {
    float acc = 0.f;
    if (vec) {
        for (int k = lane * 8; k < K; k += 256) {
            float wv[8];
            load8_as_f32(w, sizeof(T) == 4 ? QS_F32 : QS_BF16, k, wv);
            const float4 a = *reinterpret_cast<const float4*>(x + k), b = *reinterpret_cast<const float4*>(x + k + 4);
            acc = fmaf(wv[0], a.x, acc); acc = fmaf(wv[1], a.y, acc); acc = fmaf(wv[2], a.z, acc); acc = fmaf(wv[3], a.w, acc);
            acc = fmaf(wv[4], b.x, acc); acc = fmaf(wv[5], b.y, acc); acc = fmaf(wv[6], b.z, acc); acc = fmaf(wv[7], b.w, acc);
        }
    } else {
        for (int k = lane; k < K; k += 32) acc = fmaf(to_f32(w[k]), x[k], acc);
    }
    return warp_sum(acc);
}

// hidden[pair, f] = act(W_up[e][f, :] . h[token, :]) for pair = token * top + j, e = idx[pair]: a block stages the
// token's row in shared memory as 32-bit floats, a warp takes one hidden unit at a time.  `gated`: an expert's matrix holds
// F gate rows above its F up rows, and hidden = act(gate . h) * (up . h).
template <typename T>
__global__ void moe_expert_up_kernel(T* __restrict__ hidden, size_t ldh, const T* __restrict__ x, size_t ldx,
                                     const T* __restrict__ w_up, const int32_t* __restrict__ idx,
                                     const int32_t* __restrict__ tok_slot, int top, int D, int F, int rows_per_block, int act,
                                     int vec, int gated, int n_experts) {
    extern __shared__ __align__(16) float xs[];
    grid_dep_launch();
    grid_dep_wait();
    const int pair = blockIdx.x, t = pair / top;
    const int f0 = blockIdx.y * rows_per_block;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (tok_slot[t] < 0 || idx[pair] >= n_experts) {        // nobody's row, or an expert that returns its input: nothing hidden
        for (int f = f0 + threadIdx.x; f < min(F, f0 + rows_per_block); f += blockDim.x) hidden[(size_t)pair * ldh + f] = from_f32<T>(0.f);
        return;
    }
    for (int i = threadIdx.x; i < D; i += blockDim.x) xs[i] = to_f32(x[(size_t)t * ldx + i]);
    __syncthreads();
    const T* w = w_up + (size_t)idx[pair] * (gated ? 2 : 1) * F * D;
    for (int f = f0 + warp; f < min(F, f0 + rows_per_block); f += warps) {
        const float acc = warp_dot(w + (size_t)f * D, xs, D, lane, vec != 0);
        const float mul = gated ? warp_dot(w + (size_t)(F + f) * D, xs, D, lane, vec != 0) : 1.0f;
        if (lane == 0) hidden[(size_t)pair * ldh + f] = from_f32<T>(apply_activation_wide(acc, act) * mul);
    }
}

// out[t, d] = sum_j wts[t, j] * (W_down[idx[t, j]][d, :] . hidden[t * top + j, :])  (+ add[t, d] * add_scale[t]),
// 32-bit.  A block stages the token's `top` hidden rows; a warp takes one output element at a time.  A choice from
// `n_experts` on adds wts[t, j] * x[t, d] instead.
template <typename T>
__global__ void moe_expert_down_kernel(float* __restrict__ out, size_t ldo, const T* __restrict__ hidden, size_t ldh,
                                       const T* __restrict__ w_down, const int32_t* __restrict__ idx,
                                       const float* __restrict__ wts, const int32_t* __restrict__ tok_slot,
                                       const void* __restrict__ add, int add_dtype, size_t ldadd,
                                       const float* __restrict__ add_scale, int top, int D, int F, int rows_per_block,
                                       int vec, const T* __restrict__ x, size_t ldx, int n_experts) {
    extern __shared__ __align__(16) float hs[];         // [top][F]
    grid_dep_launch();
    grid_dep_wait();
    const int t = blockIdx.x;
    const int d0 = blockIdx.y * rows_per_block;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, warps = blockDim.x >> 5;
    if (tok_slot[t] < 0) {
        for (int d = d0 + threadIdx.x; d < min(D, d0 + rows_per_block); d += blockDim.x) out[(size_t)t * ldo + d] = 0.f;
        return;
    }
    for (int i = threadIdx.x; i < top * F; i += blockDim.x) {
        const int j = i / F;
        hs[i] = to_f32(hidden[((size_t)t * top + j) * ldh + (i - j * F)]);
    }
    __syncthreads();
    for (int d = d0 + warp; d < min(D, d0 + rows_per_block); d += warps) {
        float total = 0.f;
        for (int j = 0; j < top; ++j) {
            const int e = idx[(size_t)t * top + j];             // the same for the whole warp
            const float y = e < n_experts ? warp_dot(w_down + ((size_t)e * D + d) * F, hs + j * F, F, lane, vec != 0)
                                          : to_f32(x[(size_t)t * ldx + d]);
            total = fmaf(wts[(size_t)t * top + j], y, total);
        }
        if (lane == 0) {
            if (add) total = fmaf(load_as_f32(add, add_dtype, (size_t)t * ldadd + d), add_scale ? add_scale[t] : 1.0f, total);
            out[(size_t)t * ldo + d] = total;
        }
    }
}

// ----------------------------------------------------------------------------- few tokens, bfloat16, each expert's matrices read once
//
// The pairs of a step of few tokens grouped by expert inside the kernels: rows of an expert's matrix are the 16-row side of
// mma.sync products of bfloat16 numbers, its tokens the side of eight columns, both straight from memory to registers.  Every product of
// 16 starts from zero and is added with a rounded 32-bit addition, as in the decode attention.  The k's
// of a product are permuted so that a lane's 16 bytes of a row are two products' worth: lane t of a row's four takes the k's
// 8 t .. 8 t + 7 of 32, on both sides.  A column does not meet the others and K is cut in four wherever the token stands, so a
// token's result does not depend on the batch.
//
// Bound by the matrices' way from memory.  Microseconds of the two kernels (every pair reading its expert by itself, as before | now), gated
// experts of D x F, `top` per token:
//   16 of 4,096 x 1,024, 4: 1 token 87 | 38, 8: 196 | 93, 16: 323 | 97, 32: 538 | 110;  16 of 2,048 x 512, 4: 128 tokens 558 | 97
//   64 of 2,048 x 512: 32 tokens of 8: 319 | 108, of 16: 667 | 132;  256 of 2,048 x 512, 8: 1 token 65 | 27, 4: 80 | 64, 8: 122 | 99, 32: 323 | 226
// 3,000 tokens of width 2,048 with the router: all products of all experts in two launches (gemm_tc.cu) instead of one each behind a wait for
// the host: 428 -> 197 us.
constexpr int CHUNK_TOKENS = 32;                        // tokens of a block: at most this many columns of an expert

__device__ __forceinline__ uint4 piece(const __nv_bfloat16* row, int k, int K) {        // eight elements, zeros behind the end
    return row && k < K ? *reinterpret_cast<const uint4*>(row + k) : make_uint4(0u, 0u, 0u, 0u);
}

// acc[m][n] += rows of matrix m (`lo`: this lane's row of the first eight, `hi`: of the last eight) times columns of tile n, k from
// k0 to k1 (multiples of 32); U steps of 32 fetched together.  FINE, where the result is not rounded to 16 bits: products of eight and
// sums over four steps in pairs, so that the sum is as near to float64 as one of 32-bit multiply-adds.
template <int MATS, int NT, int U, bool FINE>
__device__ __forceinline__ void stream_rows(float (&acc)[MATS][NT][4], const __nv_bfloat16* const (&lo)[MATS], const __nv_bfloat16* const (&hi)[MATS],
                                            const __nv_bfloat16* const (&col)[NT], int k0, int k1, int K) {
    const int t8 = (threadIdx.x & 3) * 8;
    for (int k = k0; k < k1; k += 32 * U) {
        uint4 a[U][MATS], b[U][MATS], x[U][NT];
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int at = k + u * 32 + t8, end = min(k1, K);
#pragma unroll
            for (int m = 0; m < MATS; ++m) { a[u][m] = piece(lo[m], at, end); b[u][m] = piece(hi[m], at, end); }
#pragma unroll
            for (int n = 0; n < NT; ++n) x[u][n] = piece(col[n], at, end);
        }
        float run[FINE ? 2 : 1][MATS][NT][4];
#pragma unroll
        for (int u = 0; u < U; ++u)
#pragma unroll
            for (int m = 0; m < MATS; ++m)
#pragma unroll
                for (int n = 0; n < NT; ++n) {
                    float d0[4], d1[4], d2[4], d3[4];
                    if constexpr (FINE) {
                        mma_bf16_16x8x8(d0, a[u][m].x, b[u][m].x, x[u][n].x);
                        mma_bf16_16x8x8(d1, a[u][m].y, b[u][m].y, x[u][n].y);
                        mma_bf16_16x8x8(d2, a[u][m].z, b[u][m].z, x[u][n].z);
                        mma_bf16_16x8x8(d3, a[u][m].w, b[u][m].w, x[u][n].w);
                    } else {
                        mma_bf16_16x8x16(d0, a[u][m].x, b[u][m].x, a[u][m].y, b[u][m].y, x[u][n].x, x[u][n].y);
                        mma_bf16_16x8x16(d1, a[u][m].z, b[u][m].z, a[u][m].w, b[u][m].w, x[u][n].z, x[u][n].w);
                    }
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        if constexpr (FINE) {
                            float &r0 = run[0][m][n][e], &r1 = run[1][m][n][e];
                            const float step = (d0[e] + d1[e]) + (d2[e] + d3[e]);
                            if (u % 4 == 0) r0 = step;
                            else if (u % 4 == 1) r0 += step;
                            else if (u % 4 == 2) r1 = step;
                            else acc[m][n][e] += r0 + (r1 + step);
                        } else acc[m][n][e] += d0[e] + d1[e];
                    }
                }
    }
}

// hidden[pair, f] of 16 hidden units f of one expert, for the chunk's pairs that chose it; four warps share K.
template <int MATS, int NT>
__device__ void up_columns(__nv_bfloat16* __restrict__ hidden, size_t ldh, const __nv_bfloat16* __restrict__ x, size_t ldx, const __nv_bfloat16* __restrict__ w,
                           const int* list, int n, int top, int D, int F, int f0, int act, float* red) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const __nv_bfloat16 *lo[MATS], *hi[MATS], *col[NT];
#pragma unroll
    for (int m = 0; m < MATS; ++m) {
        lo[m] = f0 + g < F ? w + ((size_t)m * F + f0 + g) * D : nullptr;
        hi[m] = f0 + g + 8 < F ? w + ((size_t)m * F + f0 + g + 8) * D : nullptr;
    }
#pragma unroll
    for (int c = 0; c < NT; ++c) col[c] = c * 8 + g < n ? x + (size_t)(list[c * 8 + g] / top) * ldx : nullptr;
    float acc[MATS][NT][4];
#pragma unroll
    for (int m = 0; m < MATS; ++m)
#pragma unroll
        for (int c = 0; c < NT; ++c) acc[m][c][0] = acc[m][c][1] = acc[m][c][2] = acc[m][c][3] = 0.f;
    const int per = ((D + 31) / 32 + 3) / 4 * 32;
    stream_rows<MATS, NT, NT == 1 ? 4 : 2, false>(acc, lo, hi, col, warp * per, min((warp + 1) * per, (D + 31) / 32 * 32), D);
    constexpr int PITCH = NT * 8 + 1;                   // red [4 warps][MATS][16 rows][PITCH]
#pragma unroll
    for (int m = 0; m < MATS; ++m)
#pragma unroll
        for (int c = 0; c < NT; ++c)
#pragma unroll
            for (int e = 0; e < 4; ++e) red[((warp * MATS + m) * 16 + g + 8 * (e >> 1)) * PITCH + c * 8 + 2 * t + (e & 1)] = acc[m][c][e];
    __syncthreads();
    for (int e = threadIdx.x; e < 16 * n; e += blockDim.x) {
        const int r = e & 15, c = e >> 4;
        float v[MATS];
#pragma unroll
        for (int m = 0; m < MATS; ++m) {
            const float* at = red + (m * 16 + r) * PITCH + c;
            v[m] = (at[0] + at[MATS * 16 * PITCH]) + (at[2 * MATS * 16 * PITCH] + at[3 * MATS * 16 * PITCH]);
        }
        const float y = apply_activation_wide(v[0], act);
        if (f0 + r < F) hidden[(size_t)list[c] * ldh + f0 + r] = __float2bfloat16_rn(MATS == 2 ? y * v[MATS - 1] : y);
    }
    __syncthreads();
}

template <bool GATED>
__global__ void __launch_bounds__(128)
moe_up_grouped_kernel(__nv_bfloat16* __restrict__ hidden, size_t ldh, const __nv_bfloat16* __restrict__ x, size_t ldx, const __nv_bfloat16* __restrict__ w_up,
                      const int32_t* __restrict__ idx, const int32_t* __restrict__ tok_slot, int T, int top, int D, int F, int act, int n_experts) {
    constexpr int MATS = GATED ? 2 : 1;
    extern __shared__ int list[];                       // the chunk's pairs that chose this expert, in order
    __shared__ float red[4 * MATS * 16 * 33];
    __shared__ int count[4];
    grid_dep_launch();
    grid_dep_wait();
    const int f0 = blockIdx.x * 16, first = blockIdx.z * CHUNK_TOKENS * top, n_pairs = min(T - (int)blockIdx.z * CHUNK_TOKENS, CHUNK_TOKENS) * top;
    // a block per expert, or, where the chunk has fewer pairs than there are experts, per pair: the first one that chose an expert serves it
    const bool by_pair = (int)gridDim.y < n_experts;
    int e = blockIdx.y;
    if (by_pair) {
        e = e < n_pairs && tok_slot[(first + e) / top] >= 0 ? idx[first + e] : -1;
        if (e >= n_experts) e = -1;
        if (e < 0 && blockIdx.y > 0) return;
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int n = 0;
    for (int base = 0; base < n_pairs; base += 128) {
        const int p = base + threadIdx.x;
        const int mine = p < n_pairs ? idx[first + p] : -1;
        const bool live = p < n_pairs && tok_slot[(first + p) / top] >= 0;
        if (blockIdx.y == 0 && p < n_pairs && (!live || mine >= n_experts))     // nobody's row, or an expert that returns its input: nothing hidden
            for (int f = f0; f < min(F, f0 + 16); ++f) hidden[(size_t)(first + p) * ldh + f] = __float2bfloat16_rn(0.f);
        const unsigned hit = __ballot_sync(0xffffffffu, live && mine == e);
        if (lane == 0) count[warp] = __popc(hit);
        __syncthreads();
        int at = n;
        for (int q = 0; q < warp; ++q) at += count[q];
        if (hit >> lane & 1) list[at + __popc(hit & ((1u << lane) - 1))] = first + p;
        n += count[0] + count[1] + count[2] + count[3];
        __syncthreads();
    }
    if (by_pair && (n == 0 || list[0] != first + (int)blockIdx.y)) return;
    const __nv_bfloat16* w = w_up + (size_t)e * MATS * F * D;
    for (int c = 0; c < n; c += 32) {
        const int m = min(32, n - c);
        if (m <= 8) up_columns<MATS, 1>(hidden, ldh, x, ldx, w, list + c, m, top, D, F, f0, act, red);
        else if (m <= 16) up_columns<MATS, 2>(hidden, ldh, x, ldx, w, list + c, m, top, D, F, f0, act, red);
        else up_columns<MATS, 4>(hidden, ldh, x, ldx, w, list + c, m, top, D, F, f0, act, red);
    }
}

// Sixteen output elements d of a chunk's tokens: warp w takes quarter w mod 4 of K of every second (fourth) expert in use; the quarters' sums
// rest in shared memory until the tokens' choices are added up in order.  128 registers a thread (two blocks of eight warps or one of sixteen);
// the form for up to 32 tokens of one expert spills 36 bytes.
template <int NT>
__device__ void down_columns(float* __restrict__ part, const __nv_bfloat16* __restrict__ hidden, size_t ldh, const __nv_bfloat16* __restrict__ w, const int* list,
                             int n, int first, int D, int F, int d0, int quarter) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const __nv_bfloat16* const lo[1] = {d0 + g < D ? w + (size_t)(d0 + g) * F : nullptr};
    const __nv_bfloat16* const hi[1] = {d0 + g + 8 < D ? w + (size_t)(d0 + g + 8) * F : nullptr};
    const __nv_bfloat16* col[NT];
#pragma unroll
    for (int c = 0; c < NT; ++c) col[c] = c * 8 + g < n ? hidden + (size_t)(first + list[c * 8 + g]) * ldh : nullptr;
    float acc[1][NT][4];
#pragma unroll
    for (int c = 0; c < NT; ++c) acc[0][c][0] = acc[0][c][1] = acc[0][c][2] = acc[0][c][3] = 0.f;
    const int per = ((F + 31) / 32 + 3) / 4 * 32;
    stream_rows<1, NT, NT == 1 ? 8 : 4, true>(acc, lo, hi, col, quarter * per, min((quarter + 1) * per, (F + 31) / 32 * 32), F);
#pragma unroll
    for (int c = 0; c < NT; ++c)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const int at = c * 8 + 2 * t + (e & 1);
            if (at < n) part[list[at] * 16 + g + 8 * (e >> 1)] = acc[0][c][e];
        }
}

__global__ void __launch_bounds__(512)
moe_down_grouped_kernel(float* __restrict__ out, size_t ldo, const __nv_bfloat16* __restrict__ hidden, size_t ldh, const __nv_bfloat16* __restrict__ w_down,
                        const int32_t* __restrict__ idx, const float* __restrict__ wts, const int32_t* __restrict__ tok_slot, const void* __restrict__ add,
                        int add_dtype, size_t ldadd, const float* __restrict__ add_scale, int T, int top, int D, int F, const __nv_bfloat16* __restrict__ x,
                        size_t ldx, int n_experts) {
    extern __shared__ float smem[];
    const int tokens = min(T - (int)blockIdx.z * CHUNK_TOKENS, CHUNK_TOKENS), n_pairs = tokens * top, most = CHUNK_TOKENS * top;
    const int t0 = blockIdx.z * CHUNK_TOKENS, first = t0 * top, d0 = blockIdx.x * 16;
    float* part = smem;                                 // [4][pairs][16]
    int* of = reinterpret_cast<int*>(part + 4 * most * 16);    // a pair's expert (behind all others: no matrices to read)
    int* order = of + most;                             // the pairs ordered by expert
    int* start = order + most;                          // where an expert's pairs begin
    __shared__ int n_live, n_used;
    grid_dep_launch();
    grid_dep_wait();
    constexpr int NONE = 0x7fffffff;
    for (int p = threadIdx.x; p < (n_pairs + 3) / 4 * 4; p += blockDim.x) {
        const int e = p < n_pairs ? idx[first + p] : NONE;
        of[p] = e < n_experts && tok_slot[t0 + p / top] >= 0 ? e : NONE;
    }
    __syncthreads();
    for (int p = threadIdx.x; p < n_pairs; p += blockDim.x) {   // a pair's place: behind the lower experts' pairs and the earlier ones of its own
        const int e = of[p];
        int rank = 0;
        for (int q = 0; q < n_pairs; q += 4) {
            const int4 o = *reinterpret_cast<const int4*>(of + q);
            rank += (o.x < e || (o.x == e && q < p)) + (o.y < e || (o.y == e && q + 1 < p)) + (o.z < e || (o.z == e && q + 2 < p)) +
                    (o.w < e || (o.w == e && q + 3 < p));
        }
        order[rank] = p;
    }
    __syncthreads();
    if (threadIdx.x < 32) {                             // the experts in use: where one begins along `order`
        int used = 0, live = 0;
        for (int base = 0; base < n_pairs; base += 32) {
            const int r = base + threadIdx.x, e = r < n_pairs ? of[order[r]] : NONE;
            const bool opens = e != NONE && (r == 0 || of[order[r - 1]] != e);
            const unsigned open = __ballot_sync(0xffffffffu, opens);
            if (opens) start[used + __popc(open & ((1u << threadIdx.x) - 1))] = r;
            used += __popc(open);
            live += __popc(__ballot_sync(0xffffffffu, e != NONE));
        }
        if (threadIdx.x == 0) { n_used = used; n_live = live; }
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, quarter = warp & 3;
    for (int u = warp >> 2; u < n_used; u += blockDim.x >> 7) {
        const int lo = start[u], hi = u + 1 < n_used ? start[u + 1] : n_live;
        const __nv_bfloat16* w = w_down + (size_t)of[order[lo]] * D * F;
        for (int c = lo; c < hi; c += 32) {
            const int m = min(32, hi - c);
            float* mine = part + quarter * most * 16;
            if (m <= 8) down_columns<1>(mine, hidden, ldh, w, order + c, m, first, D, F, d0, quarter);
            else if (m <= 16) down_columns<2>(mine, hidden, ldh, w, order + c, m, first, D, F, d0, quarter);
            else down_columns<4>(mine, hidden, ldh, w, order + c, m, first, D, F, d0, quarter);
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < tokens * 16; e += blockDim.x) {
        const int t = e >> 4, r = e & 15, d = d0 + r;
        if (d >= D) continue;
        const size_t row = t0 + t;
        float total = 0.f;
        if (tok_slot[row] >= 0) {
            for (int j = 0; j < top; ++j) {
                const int p = t * top + j;
                float y;
                if (of[p] == NONE) y = __bfloat162float(x[row * ldx + d]);
                else {
                    const float* at = part + p * 16 + r;
                    y = (at[0] + at[most * 16]) + (at[2 * most * 16] + at[3 * most * 16]);
                }
                total = fmaf(wts[row * top + j], y, total);
            }
            if (add) total = fmaf(load_as_f32(add, add_dtype, row * ldadd + d), add_scale ? add_scale[row] : 1.0f, total);
        }
        out[row * ldo + d] = total;
    }
}

// The (token, choice) pairs ordered by expert, by one block: offsets[e] .. offsets[e + 1] are expert e's places,
// place_token[p] the token whose row goes there, pair_place[pair] the place of a pair.  Pairs of padding rows
// (slot < 0) are counted for the expert they name: their rows are zeros and nobody reads their results.
__global__ void moe_sort_kernel(int32_t* __restrict__ offsets, int32_t* __restrict__ place_token,
                                int32_t* __restrict__ pair_place, const int32_t* __restrict__ idx, int n_pairs, int top, int E) {
    __shared__ int count[MAX_EXPERTS + 1];
    grid_dep_launch();
    grid_dep_wait();
    for (int e = threadIdx.x; e <= E; e += blockDim.x) count[e] = 0;
    __syncthreads();
    constexpr int AHEAD = 4;                            // choices fetched before the first of them is counted
    for (int p0 = threadIdx.x; p0 < n_pairs; p0 += AHEAD * blockDim.x) {
        int e[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) e[i] = p0 + i * (int)blockDim.x < n_pairs ? idx[p0 + i * blockDim.x] : -1;
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) if (e[i] >= 0) atomicAdd(&count[e[i]], 1);
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        int run = 0;
        for (int e = 0; e < E; ++e) { const int c = count[e]; offsets[e] = run; count[e] = run; run += c; }
        offsets[E] = run;
    }
    __syncthreads();
    // a pair's place inside its expert's range is whatever the counter gives it: a row's products do not depend
    // on where the row lies, so the order is free
    for (int p0 = threadIdx.x; p0 < n_pairs; p0 += AHEAD * blockDim.x) {
        int e[AHEAD];
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) e[i] = p0 + i * (int)blockDim.x < n_pairs ? idx[p0 + i * blockDim.x] : -1;
#pragma unroll
        for (int i = 0; i < AHEAD; ++i) {
            if (e[i] < 0) continue;
            const int p = p0 + i * blockDim.x, place = atomicAdd(&count[e[i]], 1);
            place_token[place] = p / top;
            pair_place[p] = place;
        }
    }
}

// out[t, :] = sum_j wts[t, j] * y[pair_place[t * top + j], :]  (+ add[t, :] * add_scale[t]), in 32-bit; a place from n_rows on
// (`rows_dev`: the number read on the device) stands for the token's own input x[t, :].  VEC: four elements at a time.
template <typename TY, bool VEC>
__global__ void moe_combine_kernel(float* __restrict__ out, size_t ldo, const TY* __restrict__ y, size_t ldy,
                                   const int32_t* __restrict__ pair_place, const float* __restrict__ wts,
                                   const int32_t* __restrict__ tok_slot, const void* __restrict__ add, int add_dtype,
                                   size_t ldadd, const float* __restrict__ add_scale, int top, int D, const void* __restrict__ x,
                                   int x_dtype, size_t ldx, int n_rows, const int32_t* __restrict__ rows_dev) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t t = blockIdx.x;
    const bool live = tok_slot[t] >= 0;
    if (rows_dev) n_rows = *rows_dev;
    if (VEC) {
        for (int d = threadIdx.x * 4; d < D; d += blockDim.x * 4) {
            float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
            if (live) {
#pragma unroll 4
                for (int j = 0; j < top; ++j) {
                    const int place = pair_place[t * top + j];
                    const float w = wts[t * top + j];
                    float4 v;
                    if (place < n_rows) v = *reinterpret_cast<const float4*>(y + (size_t)place * ldy + d);
                    else v = make_float4(load_as_f32(x, x_dtype, t * ldx + d), load_as_f32(x, x_dtype, t * ldx + d + 1),
                                         load_as_f32(x, x_dtype, t * ldx + d + 2), load_as_f32(x, x_dtype, t * ldx + d + 3));
                    total.x = fmaf(w, v.x, total.x); total.y = fmaf(w, v.y, total.y); total.z = fmaf(w, v.z, total.z); total.w = fmaf(w, v.w, total.w);
                }
                if (add) {
                    const float w = add_scale ? add_scale[t] : 1.0f;
                    const size_t at = t * ldadd + d;
                    total.x = fmaf(load_as_f32(add, add_dtype, at), w, total.x); total.y = fmaf(load_as_f32(add, add_dtype, at + 1), w, total.y);
                    total.z = fmaf(load_as_f32(add, add_dtype, at + 2), w, total.z); total.w = fmaf(load_as_f32(add, add_dtype, at + 3), w, total.w);
                }
            }
            *reinterpret_cast<float4*>(out + t * ldo + d) = total;
        }
        return;
    }
    for (int d = threadIdx.x; d < D; d += blockDim.x) {
        float total = 0.f;
        if (live) {
            for (int j = 0; j < top; ++j) {
                const int place = pair_place[t * top + j];
                total = fmaf(wts[t * top + j], place < n_rows ? to_f32(y[(size_t)place * ldy + d]) : load_as_f32(x, x_dtype, t * ldx + d), total);
            }
            if (add) total = fmaf(load_as_f32(add, add_dtype, t * ldadd + d), add_scale ? add_scale[t] : 1.0f, total);
        }
        out[t * ldo + d] = total;
    }
}

}  // namespace

QS_API int qs_moe_route(int32_t* idx, float* wts, float* shared_gate, const float* z, long long ldz, const void* corr,
                        int corr_dtype, int T, int E, int top, int groups, int keep, float scale, int gate_col,
                        int score_kind, int group_kind, float renorm_eps, cudaStream_t stream) {
    if (T == 0) return QS_OK;
    QS_REQUIRE(T > 0 && E > 0 && E <= MAX_EXPERTS && top > 0 && top <= E, "moe_route: bad sizes T=%d E=%d top=%d", T, E, top);
    QS_REQUIRE(groups > 0 && E % groups == 0 && keep > 0 && keep <= groups, "moe_route: %d experts in %d groups, %d kept", E, groups, keep);
    QS_REQUIRE(keep * (E / groups) >= top, "moe_route: %d kept groups of %d experts cannot give %d choices", keep, E / groups, top);
    const int warps = 4;
    const size_t smem = (size_t)warps * (2 * E + groups) * sizeof(float);
    cudaError_t e = qs_launch_dependent(moe_route_kernel, dim3((T + warps - 1) / warps), dim3(warps * 32), smem, stream, idx, wts,
                                        shared_gate, z, (size_t)ldz, corr, corr_dtype, T, E, top, groups, keep, scale, gate_col, score_kind,
                                        group_kind, renorm_eps);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_route: %s", cudaGetErrorString(e));
    return qs_check_launch("moe_route");
}

QS_API int qs_moe_expert_up(void* hidden, long long ldh, const void* x, long long ldx, const void* w_up, int dtype,
                            const int32_t* idx, const int32_t* tok_slot, int T, int top, int D, int F, int act,
                            int gated, int n_experts, cudaStream_t stream) {
    if (T == 0) return QS_OK;
    QS_REQUIRE(T > 0 && top > 0 && D > 0 && F > 0, "moe_expert_up: bad sizes");
    QS_REQUIRE((size_t)D * sizeof(float) <= 200 * 1024, "moe_expert_up: width %d does not fit shared memory", D);
    if (dtype == QS_BF16 && D % 8 == 0 && ldx % 8 == 0 && ldh % 8 == 0 && ((uintptr_t)x % 16) == 0 && ((uintptr_t)w_up % 16) == 0 &&
        ((uintptr_t)hidden % 16) == 0 && top <= 64) {
        typedef __nv_bfloat16 bf16;
        const int pairs = (T < CHUNK_TOKENS ? T : CHUNK_TOKENS) * top;
        const dim3 blocks((F + 15) / 16, n_experts < pairs ? n_experts : pairs, (T + CHUNK_TOKENS - 1) / CHUNK_TOKENS);
        const cudaError_t err = gated
            ? qs_launch_dependent(moe_up_grouped_kernel<true>, blocks, dim3(128), CHUNK_TOKENS * top * sizeof(int), stream, (bf16*)hidden, (size_t)ldh,
                                  (const bf16*)x, (size_t)ldx, (const bf16*)w_up, idx, tok_slot, T, top, D, F, act, n_experts)
            : qs_launch_dependent(moe_up_grouped_kernel<false>, blocks, dim3(128), CHUNK_TOKENS * top * sizeof(int), stream, (bf16*)hidden, (size_t)ldh,
                                  (const bf16*)x, (size_t)ldx, (const bf16*)w_up, idx, tok_slot, T, top, D, F, act, n_experts);
        if (err != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_expert_up: %s", cudaGetErrorString(err));
        return qs_check_launch("moe_expert_up");
    }
    const int rows_per_block = 32;
    const size_t smem = (size_t)D * sizeof(float);
    const int vec = D % 8 == 0 && ((uintptr_t)w_up % 16) == 0;
    dim3 grid(T * top, (F + rows_per_block - 1) / rows_per_block);
    cudaError_t e = cudaSuccess;
#define GO(TT) do { if (smem > 48 * 1024) e = cudaFuncSetAttribute(moe_expert_up_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e == cudaSuccess) e = qs_launch_dependent(moe_expert_up_kernel<TT>, grid, dim3(256), smem, stream, (TT*)hidden, (size_t)ldh, (const TT*)x, \
        (size_t)ldx, (const TT*)w_up, idx, tok_slot, top, D, F, rows_per_block, act, vec, gated, n_experts); } while (0)
    if (dtype == QS_F32) GO(float);
    else if (dtype == QS_BF16) GO(__nv_bfloat16);
    else return qs_fail(QS_ERR_INVALID_INPUT, "moe_expert_up: unknown dtype %d", dtype);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_expert_up: %s", cudaGetErrorString(e));
    return qs_check_launch("moe_expert_up");
}

QS_API int qs_moe_expert_down(float* out, long long ldo, const void* hidden, long long ldh, const void* w_down, int dtype,
                              const int32_t* idx, const float* wts, const int32_t* tok_slot, const void* add, int add_dtype,
                              long long ldadd, const float* add_scale, int T, int top, int D, int F, const void* x, long long ldx,
                              int n_experts, cudaStream_t stream) {
    if (T == 0) return QS_OK;
    QS_REQUIRE(T > 0 && top > 0 && D > 0 && F > 0, "moe_expert_down: bad sizes");
    const size_t smem = (size_t)top * F * sizeof(float);
    QS_REQUIRE(smem <= 200 * 1024, "moe_expert_down: %d x %d hidden values do not fit shared memory", top, F);
    constexpr int MOST_CHOICES = 16;
    auto grouped = [](int choices) { return (size_t)CHUNK_TOKENS * choices * (4 * 16 + 3) * sizeof(float); };
    if (dtype == QS_BF16 && F % 8 == 0 && ldh % 8 == 0 && ((uintptr_t)hidden % 16) == 0 && ((uintptr_t)w_down % 16) == 0 && top <= MOST_CHOICES) {
        // sixteen warps to a block where the blocks leave SMs to themselves
        const int threads = (D + 15) / 16 * ((T + CHUNK_TOKENS - 1) / CHUNK_TOKENS) <= 148 ? 512 : 256;
        // the limit for the most choices, whatever these are: another thread's launch may come between it and this one's
        cudaError_t err = cudaFuncSetAttribute(moe_down_grouped_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)grouped(MOST_CHOICES));
        if (err == cudaSuccess)
            err = qs_launch_dependent(moe_down_grouped_kernel, dim3((D + 15) / 16, 1, (T + CHUNK_TOKENS - 1) / CHUNK_TOKENS), dim3(threads), grouped(top), stream, out, (size_t)ldo,
                                      (const __nv_bfloat16*)hidden, (size_t)ldh, (const __nv_bfloat16*)w_down, idx, wts, tok_slot, add, add_dtype, (size_t)ldadd, add_scale,
                                      T, top, D, F, (const __nv_bfloat16*)x, (size_t)ldx, n_experts);
        if (err != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_expert_down: %s", cudaGetErrorString(err));
        return qs_check_launch("moe_expert_down");
    }
    const int rows_per_block = 32;
    const int vec = F % 8 == 0 && ((uintptr_t)w_down % 16) == 0;
    dim3 grid(T, (D + rows_per_block - 1) / rows_per_block);
    cudaError_t e = cudaSuccess;
#define GO(TT) do { if (smem > 48 * 1024) e = cudaFuncSetAttribute(moe_expert_down_kernel<TT>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e == cudaSuccess) e = qs_launch_dependent(moe_expert_down_kernel<TT>, grid, dim3(256), smem, stream, out, (size_t)ldo, (const TT*)hidden, \
        (size_t)ldh, (const TT*)w_down, idx, wts, tok_slot, add, add_dtype, (size_t)ldadd, add_scale, top, D, F, rows_per_block, vec, (const TT*)x, (size_t)ldx, \
        n_experts); } while (0)
    if (dtype == QS_F32) GO(float);
    else if (dtype == QS_BF16) GO(__nv_bfloat16);
    else return qs_fail(QS_ERR_INVALID_INPUT, "moe_expert_down: unknown dtype %d", dtype);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_expert_down: %s", cudaGetErrorString(e));
    return qs_check_launch("moe_expert_down");
}

QS_API int qs_moe_sort(int32_t* offsets, int32_t* place_token, int32_t* pair_place, const int32_t* idx, int n_pairs,
                       int top, int E, cudaStream_t stream) {
    QS_REQUIRE(n_pairs > 0 && top > 0 && E > 0 && E <= MAX_EXPERTS, "moe_sort: bad sizes");
    const cudaError_t e = qs_launch_dependent(moe_sort_kernel, dim3(1), dim3(1024), 0, stream, offsets, place_token, pair_place, idx, n_pairs, top, E);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_sort: %s", cudaGetErrorString(e));
    return qs_check_launch("moe_sort");
}

QS_API int qs_moe_combine(float* out, long long ldo, const void* y, int y_dtype, long long ldy, const int32_t* pair_place,
                          const float* wts, const int32_t* tok_slot, const void* add, int add_dtype, long long ldadd,
                          const float* add_scale, int T, int top, int D, const void* x, int x_dtype, long long ldx, int n_rows,
                          const int32_t* rows_dev, cudaStream_t stream) {
    if (T == 0) return QS_OK;
    QS_REQUIRE(T > 0 && top > 0 && D > 0, "moe_combine: bad sizes");
    const int threads = D >= 1024 ? 256 : 128;
    cudaError_t e;
#define GO(TY, VEC) e = qs_launch_dependent(moe_combine_kernel<TY, VEC>, dim3(T), dim3(threads), 0, stream, out, (size_t)ldo, (const TY*)y, \
        (size_t)ldy, pair_place, wts, tok_slot, add, add_dtype, (size_t)ldadd, add_scale, top, D, x, x_dtype, (size_t)ldx, n_rows, rows_dev)
    if (y_dtype == QS_F32 && D % 4 == 0 && ldy % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)y % 16) == 0 && ((uintptr_t)out % 16) == 0) GO(float, true);
    else if (y_dtype == QS_F32) GO(float, false);
    else if (y_dtype == QS_BF16) GO(__nv_bfloat16, false);
    else return qs_fail(QS_ERR_INVALID_INPUT, "moe_combine: unknown dtype %d", y_dtype);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "moe_combine: %s", cudaGetErrorString(e));
    return qs_check_launch("moe_combine");
}

// The matrix products of the library (csrc/gemm_tc.cu, csrc/linear_simt.cu).
extern "C" int qs_gemm_tc(void* C, int c_dtype, const void* A, const void* W, const void* bias, int bias_dtype, int act,
                          const void* res1, const void* res2, int M, int N, int K, long long lda, long long ldw,
                          long long ldc, long long ldr, float* ws, long long ws_floats, int32_t* counters, int n_counters,
                          int32_t* status, int smem_kb, cudaStream_t stream);
extern "C" int qs_linear_simt(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                              const void* bias, int bias_dtype, int act, const void* res1, const void* res2,
                              int M, int N, int K, long long lda, long long ldc, long long ldr, float* ws, long long ws_floats,
                              cudaStream_t stream);

// One product per expert over its rows, all launched by this one call: C[rows of e] = A[rows of e] W[e]^T with
// W [E][N][K] and the experts' row ranges `offsets` (E + 1 entries, on the HOST).  `use_tc`: the tensor-core product
// (bfloat16 operands that it takes) with its scratch `ws`, `counters`, `status`; else the CUDA-core product.
//
// An expert's product is small (a thousand rows fill a sixth of the SMs with tiles), so the experts are dealt to
// EXPERT_STREAMS streams of the library's own that fork from `stream` and join it again before the call returns; each
// stream has its own share of the scratch.  While `stream` is being captured everything stays on it, in order.
namespace {
constexpr int EXPERT_STREAMS = 8, MAX_DEVICES = 16;
struct ExpertStreams { cudaStream_t side[EXPERT_STREAMS]; cudaEvent_t fork, join[EXPERT_STREAMS]; bool ready; };
ExpertStreams g_expert_streams[MAX_DEVICES];

ExpertStreams* expert_streams() {
    int device = -1;
    if (cudaGetDevice(&device) != cudaSuccess || device < 0 || device >= MAX_DEVICES) return nullptr;
    ExpertStreams& p = g_expert_streams[device];
    if (!p.ready) {
        if (cudaEventCreateWithFlags(&p.fork, cudaEventDisableTiming) != cudaSuccess) return nullptr;
        for (int i = 0; i < EXPERT_STREAMS; ++i)
            if (cudaStreamCreateWithFlags(&p.side[i], cudaStreamNonBlocking) != cudaSuccess ||
                cudaEventCreateWithFlags(&p.join[i], cudaEventDisableTiming) != cudaSuccess) return nullptr;
        p.ready = true;
    }
    return &p;
}
}  // namespace

QS_API int qs_expert_products(void* C, int c_dtype, long long ldc, const void* A, int a_dtype, long long lda, const void* W,
                              int w_dtype, const int32_t* offsets, int E, int N, int K, int use_tc, float* ws,
                              long long ws_floats, int32_t* counters, int n_counters, int32_t* status, cudaStream_t stream) {
    QS_REQUIRE(E > 0 && N > 0 && K > 0 && offsets, "expert_products: bad sizes");
    const size_t a_size = a_dtype == QS_F32 ? 4 : 2, c_size = c_dtype == QS_F32 ? 4 : 2, w_size = w_dtype == QS_F32 ? 4 : 2;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    ExpertStreams* pool = nullptr;
    if (E > 1 && cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone)
        pool = expert_streams();
    const int lanes = pool ? EXPERT_STREAMS : 1;
    const long long ws_share = ws_floats / lanes / 4 * 4;
    const int counter_share = n_counters / lanes;
    if (pool) {
        if (cudaEventRecord(pool->fork, stream) != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "expert_products: cannot fork");
        for (int i = 0; i < lanes; ++i) cudaStreamWaitEvent(pool->side[i], pool->fork, 0);
    }
    int rc = QS_OK;
    for (int e = 0; e < E && rc == QS_OK; ++e) {
        const int lo = offsets[e], M = offsets[e + 1] - lo;
        if (M <= 0) continue;
        const int lane = e % lanes;
        cudaStream_t st = pool ? pool->side[lane] : stream;
        char* c = (char*)C + (size_t)lo * ldc * c_size;
        const char* a = (const char*)A + (size_t)lo * lda * a_size;
        const char* w = (const char*)W + (size_t)e * N * K * w_size;
        rc = use_tc ? qs_gemm_tc(c, c_dtype, a, w, nullptr, 0, QS_ACT_NONE, nullptr, nullptr, M, N, K, lda, K, ldc, N,
                                 ws + (size_t)lane * ws_share, ws_share, counters + (size_t)lane * counter_share, counter_share,
                                 status, 0, st)
                    : qs_linear_simt(c, c_dtype, a, a_dtype, w, w_dtype, nullptr, 0, QS_ACT_NONE, nullptr, nullptr, M, N, K, lda,
                                     ldc, N, nullptr, 0, st);
    }
    if (pool)                                           // also after a failed launch: `stream` must not run ahead of the others
        for (int i = 0; i < lanes; ++i) {
            cudaEventRecord(pool->join[i], pool->side[i]);
            cudaStreamWaitEvent(stream, pool->join[i], 0);
        }
    return rc;
}

// One product per head over the same rows, dealt to the same streams: C[:, head h] = A[:, head h] W[h]^T with W [H][N][K],
// head h's K inputs at A + h * head_a and its N results at C + h * head_c (elements), rows `lda` and `ldc` apart.
QS_API int qs_head_products(void* C, int c_dtype, long long ldc, long long head_c, const void* A, int a_dtype, long long lda,
                            long long head_a, const void* W, int w_dtype, int M, int H, int N, int K, int use_tc, float* ws,
                            long long ws_floats, int32_t* counters, int n_counters, int32_t* status, cudaStream_t stream) {
    QS_REQUIRE(M > 0 && H > 0 && N > 0 && K > 0, "head_products: bad sizes");
    const size_t a_size = a_dtype == QS_F32 ? 4 : 2, c_size = c_dtype == QS_F32 ? 4 : 2, w_size = w_dtype == QS_F32 ? 4 : 2;
    cudaStreamCaptureStatus capturing = cudaStreamCaptureStatusNone;
    ExpertStreams* pool = nullptr;
    if (H > 1 && cudaStreamIsCapturing(stream, &capturing) == cudaSuccess && capturing == cudaStreamCaptureStatusNone)
        pool = expert_streams();
    const int lanes = pool ? EXPERT_STREAMS : 1;
    const long long ws_share = ws_floats / lanes / 4 * 4;
    const int counter_share = n_counters / lanes;
    if (pool) {
        if (cudaEventRecord(pool->fork, stream) != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "head_products: cannot fork");
        for (int i = 0; i < lanes; ++i) cudaStreamWaitEvent(pool->side[i], pool->fork, 0);
    }
    int rc = QS_OK;
    for (int h = 0; h < H && rc == QS_OK; ++h) {
        const int lane = h % lanes;
        cudaStream_t st = pool ? pool->side[lane] : stream;
        char* c = (char*)C + (size_t)h * head_c * c_size;
        const char* a = (const char*)A + (size_t)h * head_a * a_size;
        const char* w = (const char*)W + (size_t)h * N * K * w_size;
        rc = use_tc ? qs_gemm_tc(c, c_dtype, a, w, nullptr, 0, QS_ACT_NONE, nullptr, nullptr, M, N, K, lda, K, ldc, N,
                                 ws + (size_t)lane * ws_share, ws_share, counters + (size_t)lane * counter_share, counter_share,
                                 status, 0, st)
                    : qs_linear_simt(c, c_dtype, a, a_dtype, w, w_dtype, nullptr, 0, QS_ACT_NONE, nullptr, nullptr, M, N, K, lda,
                                     ldc, N, nullptr, 0, st);
    }
    if (pool)
        for (int i = 0; i < lanes; ++i) {
            cudaEventRecord(pool->join[i], pool->side[i]);
            cudaStreamWaitEvent(stream, pool->join[i], 0);
        }
    return rc;
}
