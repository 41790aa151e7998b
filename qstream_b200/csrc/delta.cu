// What a gated delta rule needs between its projections and its scan.
//
// q, k (G heads of dk) and v (H heads of dv) each pass a short causal convolution over time per channel
// (taps [channels, n]: tap n - 1 weighs the token itself, tap n - 1 - j the token j places back, and what lies before a
// sequence counts as zero) and silu; q and k then become unit vectors per head, x / sqrt(sum x^2 + unit_eps), q also
// times q_scale.  The decay per token, head
// and key channel is g = exp(-exp(A_log_h) * softplus(a)), the step size per token and head beta = sigmoid(b).
// Everything is 32-bit and leaves in 32-bit: these values enter the recurrence.
//
// The convolution's last n - 1 inputs of a sequence are state: [slots][n - 1][C] in the inputs' type, channels in
// the order q | k | v, row n - 2 the newest, zero when the slot is taken.  `delta_prepare_kernel` reads it for the
// tokens whose predecessors came in earlier steps; `conv_state_update_kernel` runs after it and leaves the last
// n - 1 inputs of what the slot held and the step brought.
#include "group_norm.cuh"

namespace {

constexpr int MAX_TAPS = 8;

template <typename TI>
__global__ void delta_prepare_kernel(float* __restrict__ qo, float* __restrict__ ko, float* __restrict__ vo,
                                     float* __restrict__ go, float* __restrict__ bo,
                                     const TI* __restrict__ q, const TI* __restrict__ k, const TI* __restrict__ v, size_t ldp,
                                     const void* __restrict__ wq, const void* __restrict__ wk, const void* __restrict__ wv,
                                     int w_dtype, int taps, const TI* __restrict__ conv_state, size_t slot_stride,
                                     const float* __restrict__ a, size_t lda, const float* __restrict__ bl, size_t ldb,
                                     const void* __restrict__ a_log, int a_log_dtype,
                                     const int32_t* __restrict__ tok_slot, const int32_t* __restrict__ tok_pos,
                                     int G, int H, int dk, int dv, float q_scale, float unit_eps) {
    extern __shared__ float x_of[];                     // [C] the token's channels after convolution and silu
    __shared__ float inv_norm[64];                      // per head of q and k, in rounds of 64
    grid_dep_launch();
    grid_dep_wait();
    const int t = blockIdx.x;
    const int nq = G * dk, nv = H * dv, C = 2 * nq + nv;
    const int slot = tok_slot[t];
    if (slot < 0) {                                     // a row that belongs to nobody
        for (int c = threadIdx.x; c < nq; c += blockDim.x) { qo[(size_t)t * nq + c] = 0.f; ko[(size_t)t * nq + c] = 0.f; }
        for (int c = threadIdx.x; c < nv; c += blockDim.x) vo[(size_t)t * nv + c] = 0.f;
        for (int c = threadIdx.x; c < H * dk; c += blockDim.x) go[(size_t)t * H * dk + c] = 1.f;
        for (int c = threadIdx.x; c < H; c += blockDim.x) bo[(size_t)t * H + c] = 0.f;
        return;
    }
    const int pos = tok_pos[t];
    // how many of the token's predecessors came with this step (they lie in the rows just above), up to taps - 1
    int here = 0;
    while (here < taps - 1 && t - here - 1 >= 0 && tok_slot[t - here - 1] == slot && tok_pos[t - here - 1] == pos - here - 1) ++here;
    const TI* held = conv_state + (size_t)slot * slot_stride;
    for (int c = threadIdx.x; c < C; c += blockDim.x) {
        const TI* src; const void* w; int ch;
        if (c < nq) { src = q; w = wq; ch = c; }
        else if (c < 2 * nq) { src = k; w = wk; ch = c - nq; }
        else { src = v; w = wv; ch = c - 2 * nq; }
        float acc = 0.f;
        for (int j = 0; j < taps; ++j) {                // the input j tokens back meets tap number taps - 1 - j
            float x;
            if (j <= here) x = to_f32(src[(size_t)(t - j) * ldp + ch]);
            else x = to_f32(held[(size_t)(taps - 1 - (j - here)) * C + c]);
            acc = fmaf(load_as_f32(w, w_dtype, (size_t)ch * taps + taps - 1 - j), x, acc);
        }
        x_of[c] = silu_f32(acc);
    }
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
    for (int first = 0; first < 2 * G; first += 64) {   // the heads of q, then those of k
        const int n = min(64, 2 * G - first);
        for (int hd = warp; hd < n; hd += warps) {
            const float* x = x_of + (size_t)(first + hd) * dk;
            float sq = 0.f;
            for (int i = lane; i < dk; i += 32) sq = fmaf(x[i], x[i], sq);
            sq = warp_sum(sq);
            if (lane == 0) inv_norm[hd] = 1.0f / sqrtf(sq + unit_eps);
        }
        __syncthreads();
        for (int e = threadIdx.x; e < n * dk; e += blockDim.x) {
            const int hd = first + e / dk, i = e % dk;
            const float val = x_of[(size_t)hd * dk + i] * inv_norm[e / dk];
            if (hd < G) qo[(size_t)t * nq + (size_t)hd * dk + i] = val * q_scale;
            else ko[(size_t)t * nq + (size_t)(hd - G) * dk + i] = val;
        }
        __syncthreads();
    }
    for (int c = threadIdx.x; c < nv; c += blockDim.x) vo[(size_t)t * nv + c] = x_of[2 * nq + c];
    for (int c = threadIdx.x; c < H * dk; c += blockDim.x) {
        const float rate = expf(load_as_f32(a_log, a_log_dtype, c / dk));
        go[(size_t)t * H * dk + c] = expf(-rate * softplus_f32(a[(size_t)t * lda + c]));
    }
    for (int c = threadIdx.x; c < H; c += blockDim.x) bo[(size_t)t * H + c] = sigmoid_f32(bl[(size_t)t * ldb + c]);
}

// The same with eight neighbouring channels per thread, from the loads to the stores in registers: the heads' sums by shuffles over the
// dk / 8 lanes of a head (a power of two), 16-byte pieces throughout.  The blocks of a token share its pieces; the decays' follow the
// channels'.  Bound by instruction issue (silu, softplus and two exponentials per element, all in full precision).  2,000 tokens of
// 4,096 channels and 2,048 decays: 37 us, a channel at a time 91 us.
template <typename TI, int TAPS>
__global__ void __launch_bounds__(256)
delta_prepare_pieces_kernel(float* __restrict__ qo, float* __restrict__ ko, float* __restrict__ vo, float* __restrict__ go, float* __restrict__ bo,
                            const TI* __restrict__ q, const TI* __restrict__ k, const TI* __restrict__ v, size_t ldp, const TI* __restrict__ wq,
                            const TI* __restrict__ wk, const TI* __restrict__ wv, const TI* __restrict__ conv_state, size_t slot_stride,
                            const float* __restrict__ a, size_t lda, const float* __restrict__ bl, size_t ldb, const void* __restrict__ a_log,
                            int a_log_dtype, const int32_t* __restrict__ tok_slot, const int32_t* __restrict__ tok_pos, int G, int H, int dk, int dv,
                            float q_scale, float unit_eps) {
    constexpr int CODE = sizeof(TI) == 4 ? QS_F32 : QS_BF16;
    grid_dep_launch();
    grid_dep_wait();
    const size_t t = blockIdx.x;
    const int nq = G * dk, nv = H * dv, C = 2 * nq + nv, conv = C / 8, all = conv + H * dk / 8, lanes = dk / 8;
    const int slot = tok_slot[t], pos = tok_pos[t];
    int here = 0;                                       // predecessors that came with this step, up to TAPS - 1
    while (here < TAPS - 1 && (int)t - here - 1 >= 0 && tok_slot[t - here - 1] == slot && tok_pos[t - here - 1] == pos - here - 1) ++here;
    const TI* held = conv_state + (size_t)max(slot, 0) * slot_stride;
    // whole warps go round together: the pieces of a head are neighbouring lanes of one warp
    for (int base = blockIdx.y * blockDim.x; base < all; base += gridDim.y * blockDim.x) {
        const int p = base + threadIdx.x;
        if (p < conv) {
            const int c = p * 8;
            const bool of_q = c < nq, of_k = !of_q && c < 2 * nq;
            const TI* src = of_q ? q + c : of_k ? k + (c - nq) : v + (c - 2 * nq);
            const TI* w = of_q ? wq + (size_t)c * TAPS : of_k ? wk + (size_t)(c - nq) * TAPS : wv + (size_t)(c - 2 * nq) * TAPS;
            float* dst = of_q ? qo + t * nq + c : of_k ? ko + t * nq + (c - nq) : vo + t * nv + (c - 2 * nq);
            float y[8], x[TAPS][8], wt[TAPS][8];
            if (slot >= 0) {
#pragma unroll
                for (int j = 0; j < TAPS; ++j) {
                    load8_as_f32(j <= here ? src + (t - j) * ldp : held + (size_t)(TAPS - 1 - (j - here)) * C + c, CODE, 0, x[j]);
                    load8_as_f32(w + 8 * j, CODE, 0, wt[j]);    // element e of the eight channels' taps: channel e / TAPS, tap e % TAPS
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    float acc = 0.f;
#pragma unroll
                    for (int j = 0; j < TAPS; ++j) {
                        const int e = i * TAPS + TAPS - 1 - j;
                        acc = fmaf(wt[e / 8][e % 8], x[j][i], acc);
                    }
                    y[i] = silu_f32(acc);
                }
            } else {                                    // a row that belongs to nobody
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = 0.f;
            }
            // (the heads of q and k fill whole groups of lanes, so these take part together)
            if (c < 2 * nq) {
                float sq = 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) sq = fmaf(y[i], y[i], sq);
                const unsigned mask = lanes == 32 ? 0xffffffffu : ((1u << lanes) - 1) << (threadIdx.x & 31 & ~(lanes - 1));
                for (int o = lanes / 2; o > 0; o >>= 1) sq += __shfl_xor_sync(mask, sq, o);
                const float inv = slot >= 0 ? 1.0f / sqrtf(sq + unit_eps) : 0.f;
#pragma unroll
                for (int i = 0; i < 8; ++i) { y[i] *= inv; if (of_q) y[i] *= q_scale; }
            }
            store8(dst, y);
        } else if (p < all) {
            const int c = (p - conv) * 8;
            float y[8];
            if (slot >= 0) {
                load8_as_f32(a + t * lda, QS_F32, c, y);
                const float rate = expf(load_as_f32(a_log, a_log_dtype, c / dk));
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = expf(-rate * softplus_f32(y[i]));
            } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) y[i] = 1.f;
            }
            store8(go + t * H * dk + c, y);
        }
    }
    if (blockIdx.y == 0)
        for (int c = threadIdx.x; c < H; c += blockDim.x) bo[t * H + c] = slot >= 0 ? sigmoid_f32(bl[t * ldb + c]) : 0.f;
}

template <typename TI>
__global__ void conv_state_update_kernel(TI* __restrict__ conv_state, size_t slot_stride, const TI* __restrict__ q,
                                         const TI* __restrict__ k, const TI* __restrict__ v, size_t ldp, int nq, int nv,
                                         int taps, const int32_t* __restrict__ seq_start,
                                         const int32_t* __restrict__ seq_slot) {
    grid_dep_launch();
    grid_dep_wait();
    const int s = blockIdx.x;
    const int slot = seq_slot[s];
    const int t0 = seq_start[s], n = seq_start[s + 1] - t0;
    if (slot < 0 || n <= 0) return;
    const int C = 2 * nq + nv, keep = taps - 1;
    TI* held = conv_state + (size_t)slot * slot_stride;
    for (int c = blockIdx.y * blockDim.x + threadIdx.x; c < C; c += gridDim.y * blockDim.x) {
        const TI* src; int ch;
        if (c < nq) { src = q; ch = c; }
        else if (c < 2 * nq) { src = k; ch = c - nq; }
        else { src = v; ch = c - 2 * nq; }
        // row j of the new state is the input n - keep + j rows into the step, or, before the step, what row j + n
        // held: rows are taken in rising order, so a row is read before this thread overwrites it
        for (int j = 0; j < keep; ++j) {
            const int idx = n - keep + j;
            held[(size_t)j * C + c] = idx >= 0 ? src[(size_t)(t0 + idx) * ldp + ch] : held[(size_t)(j + n) * C + c];
        }
    }
}

}  // namespace

// q, k, v: three column ranges of one product's result (row stride ldp, type `dtype`); a [T, H * dk] and bl [T, H]
// float32; conv_state [slots][taps - 1][2 G dk + H dv] of type `dtype`.  Outputs float32, contiguous rows.
QS_API int qs_delta_prepare(float* qo, float* ko, float* vo, float* go, float* bo, const void* q, const void* k, const void* v,
                            long long ldp, int dtype, const void* wq, const void* wk, const void* wv, int w_dtype, int taps,
                            const void* conv_state, long long slot_stride, const float* a, long long lda, const float* bl,
                            long long ldb, const void* a_log, int a_log_dtype, const int32_t* tok_slot,
                            const int32_t* tok_pos, int T_rows, int G, int H, int dk, int dv, float q_scale, float unit_eps,
                            cudaStream_t stream) {
    if (T_rows == 0) return QS_OK;
    QS_REQUIRE(T_rows > 0 && G > 0 && H > 0 && dk > 0 && dv > 0, "delta_prepare: bad sizes");
    QS_REQUIRE(taps >= 1 && taps <= MAX_TAPS, "delta_prepare: %d taps (1 to %d)", taps, MAX_TAPS);
    QS_REQUIRE(taps == 1 || conv_state, "delta_prepare: a convolution without its state");
    const size_t smem = (size_t)(2 * G * dk + H * dv) * sizeof(float);
    QS_REQUIRE(smem <= 200 * 1024, "delta_prepare: %d channels above the shared memory of a block", 2 * G * dk + H * dv);
    const int threads = 256;
    cudaError_t e;
    // Pieces of eight channels where every row and weight begins on a piece, a head is a power of two of one warp's lanes, and the taps
    // are as many as are unrolled; from 512 tokens on a block per token fills the GPU, below that a token's pieces go to several blocks.  No
    // more threads than pieces: 2,000 float32 tokens of 96 pieces take 11.9 us, 21.4 in blocks of 256 (a channel at a time 15.8).
    const int lanes = dk / 8;
    auto fits = [&](const void* ptr) { return ((uintptr_t)ptr % 32) == 0 || (dtype == QS_BF16 && ((uintptr_t)ptr % 16) == 0); };
    if (dtype == w_dtype && taps >= 2 && taps <= 4 && dk % 8 == 0 && lanes <= 32 && (lanes & (lanes - 1)) == 0 && dv % 8 == 0 && ldp % 8 == 0 && lda % 8 == 0 &&
        slot_stride % 8 == 0 && fits(q) && fits(k) && fits(v) && fits(wq) && fits(wk) && fits(wv) && fits(conv_state) && ((uintptr_t)a % 16) == 0 &&
        ((uintptr_t)qo % 16) == 0 && ((uintptr_t)ko % 16) == 0 && ((uintptr_t)vo % 16) == 0 && ((uintptr_t)go % 16) == 0) {
        const int pieces = (2 * G * dk + H * dv + H * dk) / 8, by = T_rows >= 512 ? 1 : (pieces + 255) / 256, threads = pieces < 256 ? (pieces + 31) / 32 * 32 : 256;
#define GOP(TI, TAPS) e = qs_launch_dependent(delta_prepare_pieces_kernel<TI, TAPS>, dim3(T_rows, by), dim3(threads), 0, stream, qo, ko, vo, go, bo, (const TI*)q, \
        (const TI*)k, (const TI*)v, (size_t)ldp, (const TI*)wq, (const TI*)wk, (const TI*)wv, (const TI*)conv_state, (size_t)slot_stride, a, (size_t)lda, bl, \
        (size_t)ldb, a_log, a_log_dtype, tok_slot, tok_pos, G, H, dk, dv, q_scale, unit_eps)
#define GOT(TI) do { if (taps == 2) GOP(TI, 2); else if (taps == 3) GOP(TI, 3); else GOP(TI, 4); } while (0)
        if (dtype == QS_F32) GOT(float);
        else if (dtype == QS_BF16) GOT(__nv_bfloat16);
        else return qs_fail(QS_ERR_INVALID_INPUT, "delta_prepare: unknown dtype %d", dtype);
#undef GOT
#undef GOP
        if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "delta_prepare: %s", cudaGetErrorString(e));
        return qs_check_launch("delta_prepare");
    }
#define GO(TI) do { e = smem > 48 * 1024 ? cudaFuncSetAttribute(delta_prepare_kernel<TI>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) \
                                          : cudaSuccess; \
    if (e == cudaSuccess) e = qs_launch_dependent(delta_prepare_kernel<TI>, dim3(T_rows), dim3(threads), smem, stream, qo, ko, vo, go, bo, \
        (const TI*)q, (const TI*)k, (const TI*)v, (size_t)ldp, wq, wk, wv, w_dtype, taps, (const TI*)conv_state, (size_t)slot_stride, \
        a, (size_t)lda, bl, (size_t)ldb, a_log, a_log_dtype, tok_slot, tok_pos, G, H, dk, dv, q_scale, unit_eps); } while (0)
    if (dtype == QS_F32) GO(float);
    else if (dtype == QS_BF16) GO(__nv_bfloat16);
    else return qs_fail(QS_ERR_INVALID_INPUT, "delta_prepare: unknown dtype %d", dtype);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "delta_prepare: %s", cudaGetErrorString(e));
    return qs_check_launch("delta_prepare");
}

QS_API int qs_conv_state_update(void* conv_state, long long slot_stride, const void* q, const void* k, const void* v,
                                long long ldp, int dtype, int nq, int nv, int taps, const int32_t* seq_start,
                                const int32_t* seq_slot, int n_seq, cudaStream_t stream) {
    if (n_seq == 0 || taps <= 1) return QS_OK;
    QS_REQUIRE(n_seq > 0 && nq > 0 && nv > 0 && taps <= MAX_TAPS, "conv_state_update: bad sizes");
    const int C = 2 * nq + nv, threads = 256;
    dim3 grid(n_seq, (C + threads - 1) / threads);
    cudaError_t e;
    if (dtype == QS_F32)
        e = qs_launch_dependent(conv_state_update_kernel<float>, grid, dim3(threads), 0, stream, (float*)conv_state,
                                (size_t)slot_stride, (const float*)q, (const float*)k, (const float*)v, (size_t)ldp, nq, nv, taps,
                                seq_start, seq_slot);
    else if (dtype == QS_BF16)
        e = qs_launch_dependent(conv_state_update_kernel<__nv_bfloat16>, grid, dim3(threads), 0, stream,
                                (__nv_bfloat16*)conv_state, (size_t)slot_stride, (const __nv_bfloat16*)q, (const __nv_bfloat16*)k,
                                (const __nv_bfloat16*)v, (size_t)ldp, nq, nv, taps, seq_start, seq_slot);
    else return qs_fail(QS_ERR_INVALID_INPUT, "conv_state_update: unknown dtype %d", dtype);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "conv_state_update: %s", cudaGetErrorString(e));
    return qs_check_launch("conv_state_update");
}
