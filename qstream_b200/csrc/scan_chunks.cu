// The matrix-state recurrences of recurrent.cu over long prompts: chunks of up to 64 tokens as matrix products.
//
// Within a chunk that starts from the state S0 (a column of S per value dim, channels i of the keys)
//       o_t = (q_t * cum_t)^T S0 + sum_{j <= t} P[t][j] v_j,      P[t][j] = b_j sum_i q_t[i] k_j[i] (a_{j+1} .. a_t)[i],
//       S_end = diag(a_1 .. a_n) S0 + sum_j b_j (a_{j+1} .. a_n * k_j) v_j^T,        cum_t = a_1 .. a_t,
// with a the decays (one number per token and head, or one per token and key channel) and b the input weights.  Three kernels
// take a prompt's chunks side by side:
//   added_state_kernel      what each chunk adds to the state it starts from, and its decays
//   chunk_prefix_kernel     (recurrent.cu) the state each chunk starts from, and the sequence's last one
//   tile_output_kernel, channel_output_kernel     every token's o, written once: one decay per head, one per key channel
// Decays enter as products of at most 64 factors up to one, never as quotients, so small ones cost no precision: per token and head by a
// recursion from a token back over the earlier ones; per channel in blocks of 16 tokens, a block's own pairs walked in order, pairs of blocks
// through the products up to the blocks' common edge.
//
// The products of 32-bit numbers run on tcgen05 as products of bfloat16 terms (terms.cuh), in runs of 64 whose sums are added outside; against
// float64 they are nearer than the multiply-adds that stood here before (o, 2-norm: state-space form 1.4e-7 instead of 1.5e-7, gated memory
// 1.4e-7 instead of 1.9e-7; decay per head, over 900 tokens, 1.4e-7 instead of 3.4e-7).  q, k and v that come as bfloat16 are one term: q k^T is then one product instead
// of six.  Bound by each block's chain of fetch, split, barrier, MMAs and stores at two blocks per SM, one for what chunks add under a decay per channel with float32 operands (117 KB of
// tiles and decays; leaving out the MMAs: 63 of 76 us
// for the outputs, 42 of 47 for what the chunks add, at 4,096 tokens of 16 heads of 128 x 128, float32 operands); the split needs half of
// the issue slots.  On mma.sync the same products took 138 and 59 us, multiply-adds 139 and 66.
//
// Microseconds of the scan alone (multiply-adds | now; caches flushed): decay per head, 4,096 tokens, 16 heads of 128 x 128, float32: 236 | 150; 1,000
// tokens, bfloat16: 85 | 38; state-space form, 2,048 tokens, 64 heads of 128 x 64: 237 | 134; gated memory, 1,000 tokens, 4 heads of 256 x 256:
// 136 | 79; per channel, 3,401 tokens, 16 heads of 64 x 128: 175 | 140, 600 tokens, float32: 103 | 58; wkv, 1,000 tokens, 16 of 64 x 64: 60 | 50.
#include "scan.cuh"
#include "scan_tiles.cuh"
#include "term_tiles.cuh"

namespace {

struct Scan {
    const void *q, *k, *v;
    size_t ldq, ldk, ldv;
    const float *dlog; size_t ldd;                      // per channel: logits of the decays
    float* factors;                                     // and, from the first kernel on, the decays themselves [T_rows][H dk]
    const float *head_decay;                            // one decay per head
    const float *ga, *gb; size_t ldg;                   // per token and head: decays (less one in mode 5), input weights
    const void* bonus; int bonus_dtype;
    const int32_t* chunk_start;
    float *chunk_state, *chunk_decay;                   // [chunks][H][dk][dvp], [chunks][H][dk]
    float* o; size_t ldo;
    int H, dk, dv, dvp, qk_group, n_chunks, T_rows;       // dvp: dv rounded up to a multiple of four
    float q_scale, decay_scale;
    int vec_q, vec_k, vec_v, vec_d;                     // whether rows may be read in pieces of four
    int32_t* status;                                    // receives a code if a bounded wait ran out
};

template <int MODE>
__device__ __forceinline__ float channel_decay(float z, float scale) { return MODE == 1 ? expf(-expf(z)) : expf(log_sigmoid_f32(z) * scale); }

// The decay of channel i of head h at row t, as a factor (mode 5: less one).
template <int MODE>
__device__ __forceinline__ float decay_at(const Scan& p, size_t t, int h, int i) {
    if (MODE == 0) return p.head_decay[h];
    if (MODE == 2 || MODE == 5) return p.ga[t * p.ldg + h];
    return channel_decay<MODE>(p.dlog[t * p.ldd + (size_t)h * p.dk + i], p.decay_scale);
}
template <int MODE>
__device__ __forceinline__ float times_decay(float x, float a) { return MODE == 5 ? fmaf(x, a, x) : x * a; }

// One decay per head: its powers in 64 bits, rounded once.  The roundings of a walk over the chunk's tokens are the same in every chunk, so that they add up
// over a prompt: the state after 900 tokens, 16 heads, 3.6e-7 of its norm from 64 bits with the walk (operands above zero 4.0e-7), 1.0e-7 (0.7e-7) with
// these; by squaring in 32 bits 6.0e-7.
__device__ __forceinline__ float decay_power(float a, int n) {      // n up to 64
    double r = 1.0, b = a;
#pragma unroll
    for (int e = 0; e < 7; ++e, b *= b) if (n >> e & 1) r *= b;
    return (float)r;
}

// A chunk of more than 64 tokens (the callers cut none): this block's columns of the state walked in order in global memory.
template <typename TI, int MODE>
__device__ void walk_in_order(const Scan& p, float* __restrict__ S, int c, int h, int col0, int cols, bool output) {
    constexpr bool ONES = MODE == 2, WKV = MODE == 1;
    const int t0 = p.chunk_start[c], t1 = p.chunk_start[c + 1], hq = h / p.qk_group, dvv = ONES ? p.dv - 1 : p.dv;
    for (int col = col0 + (int)threadIdx.x; col < col0 + cols; col += blockDim.x) {
        for (int t = t0; t < t1; ++t) {
            const TI* qr = (const TI*)p.q + (size_t)t * p.ldq + hq * p.dk;
            const TI* kr = (const TI*)p.k + (size_t)t * p.ldk + hq * p.dk;
            const float v = ONES && col == dvv ? 1.f : to_f32(((const TI*)p.v)[(size_t)t * p.ldv + (size_t)h * dvv + col]);
            const float b = MODE == 2 || MODE == 5 ? p.gb[(size_t)t * p.ldg + h] : 1.f;
            float o = 0.f;
            for (int i = 0; i < p.dk; ++i) {
                const float q = to_f32(qr[i]) * (WKV ? 1.f : p.q_scale);
                const float kv = to_f32(kr[i]) * b * v, a = decay_at<MODE>(p, t, h, i);
                float* s = S + (size_t)i * p.dvp + col;
                const float before = *s, after = times_decay<MODE>(before, a) + kv;
                o = fmaf(q, WKV ? fmaf(load_as_f32(p.bonus, p.bonus_dtype, (size_t)h * p.dk + i), kv, before) : after, o);
                *s = after;
            }
            if (output) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + col] = o;
        }
    }
}

constexpr int TILE_THREADS = 256;                       // eight warps: a quarter of the TMEM lanes each, two halves of the columns

// ----------------------------------------------------------------------------- what a chunk adds

// The sum of channel i over the chunk's tokens, from the last back, by multiply-adds; `v_at` < 0: of values that are all one.  `s_w`: the tokens' weights and
// decays behind them, where there is one decay per head.
template <typename TI, int MODE>
__device__ __noinline__ float plain_added(const Scan& p, int h, int i, int t0, int n, long long v_at, const float* s_w) {
    const TI* k = (const TI*)p.k + (size_t)t0 * p.ldk + (size_t)(h / p.qk_group) * p.dk + i;
    float sum = 0.f, run = 1.f;
    for (int j = n - 1; j >= 0; --j) {
        const float v = v_at < 0 ? 1.f : to_f32(((const TI*)p.v)[(size_t)(t0 + j) * p.ldv + v_at]);
        sum = fmaf(to_f32(k[(size_t)j * p.ldk]) * (MODE == 1 || MODE == 4 ? run : s_w[j]), v, sum);
        if (MODE == 1 || MODE == 4) run *= decay_at<MODE>(p, t0 + j, h, i);
    }
    return sum;
}
// The sums of a column whose operands the terms did not hold.
template <typename TI, int MODE>
__device__ __noinline__ void mend_added(const Scan& p, float* to, int rows, int h, int i, int t0, int n, long long v_at, const float* s_w) {
    for (int x = 0; x < rows; ++x)
        if (!held(to[(size_t)x * p.dvp])) to[(size_t)x * p.dvp] = plain_added<TI, MODE>(p, h, i + x, t0, n, v_at, s_w);
}

template <typename TI> constexpr int added_smem() { return 1024 + (3 + (sizeof(TI) == 2 ? 1 : 3)) * 2 * TILE; }

// A block takes 128 value columns of one head's state, up to 128 key channels at a time: added[i][col] = sum_j kw_j[i] v_j[col], the
// tokens on the sum's side, kw_j = b_j k_j times the decays behind token j.  kw in three terms, v in VT (one where it comes as bfloat16).
// Columns on the TMEM lanes, so that a warp writes 32 neighbouring ones.
//
// Three blocks per SM for the state-space form in bfloat16 (2,048 tokens of 64 heads of 128 x 64: 64 -> 56 us); in the other forms they were slower
// (gated memory, 1,000 tokens: 79 -> 97 us for the scan; decay per head 38 -> 40).
template <typename TI, int MODE>
__global__ void __launch_bounds__(TILE_THREADS, sizeof(TI) == 2 && MODE == 5 ? 3 : 2)
added_state_kernel(const __grid_constant__ Scan p) {
    constexpr bool PER_CHANNEL = MODE == 1 || MODE == 4, ONES = MODE == 2;
    constexpr int VT = sizeof(TI) == 2 ? 1 : 3, COLS = 128, NK = CT * 16 / TILE_THREADS, NV = 2 * NK;
    constexpr uint32_t TERM = 2 * TILE, TMEM = 128;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(16) float s_a[CT], s_w[CT], part[4 * 64];
    __shared__ float s_whole;
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_slot;
    const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (tid == 0) { mbar_init(&done, 1); mbar_fence_init(); }
    if (warp == 0) { tmem_alloc(&tmem_slot, TMEM); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem = tmem_slot, tk = (smem_u32(smem_raw) + 1023) & ~1023u, tv = tk + 3 * TERM;      // [3][2 halves of 128 channels][tokens], [VT][2][tokens]
    const int col0 = blockIdx.z * COLS;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.qk_group;
    const int dvv = ONES ? p.dv - 1 : p.dv, nv = min(COLS, dvv - col0);
    float* added = p.chunk_state + ((size_t)c * p.H + h) * p.dk * p.dvp;
    float* decays = p.chunk_decay + ((size_t)c * p.H + h) * p.dk;
    auto leave = [&]() {
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, TMEM);
    };
    if (n > CT) {
        const int cols = col0 == 0 && ONES ? nv + 1 : nv;
        for (int e = tid; e < cols * p.dk; e += TILE_THREADS) added[(size_t)(e % p.dk) * p.dvp + (e / p.dk < nv ? col0 + e / p.dk : dvv)] = 0.f;
        __syncthreads();
        walk_in_order<TI, MODE>(p, added, c, h, col0, nv, false);
        if (ONES && col0 == 0) walk_in_order<TI, MODE>(p, added, c, h, dvv, 1, false);
        if (col0 == 0)
            for (int i = tid; i < p.dk; i += TILE_THREADS) {
                float a = 1.f;
                for (int t = t0; t < t0 + n; ++t) a = times_decay<MODE>(a, decay_at<MODE>(p, t, h, i));
                decays[i] = a;
            }
        leave();
        return;
    }
    Raw4<TI> rk[NK], rv[NV];
    auto fetch_k = [&](int i0) {
#pragma unroll
        for (int x = 0; x < NK; ++x) {
            const int e = tid + x * TILE_THREADS, j = e >> 4;
            get_four(rk[x], (const TI*)p.k + (size_t)(t0 + j) * p.ldk + hq * p.dk + i0, (e & 15) * 4, min(64, p.dk - i0), j < n, p.vec_k);
        }
    };
    fetch_k(0);
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const int e = tid + x * TILE_THREADS, j = e >> 5;
        get_four(rv[x], (const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)h * dvv + col0, (e & 31) * 4, nv, j < n, p.vec_v);
    }
    if (!PER_CHANNEL) {
        if (tid < CT) {
            s_a[tid] = tid < n ? decay_at<MODE>(p, t0 + tid, h, 0) : (MODE == 5 ? 0.f : 1.f);
            s_w[tid] = (MODE == 2 || MODE == 5) && tid < n ? p.gb[(size_t)(t0 + tid) * p.ldg + h] : 1.f;
        }
        __syncthreads();
        if (tid < CT) {                                 // the decays behind token tid, and its weight
            float w = 1.f;
            if constexpr (MODE == 0) {
                w = decay_power(s_a[0], max(0, n - 1 - tid));
                if (tid == 0) s_whole = decay_power(s_a[0], n);
            } else {
#pragma unroll 8
                for (int t = CT - 1; t > 0; --t) if (t > tid) w = times_decay<MODE>(w, s_a[t]);
                if (tid == 0) s_whole = times_decay<MODE>(w, s_a[0]);
            }
            s_w[tid] *= w;
        }
        __syncthreads();
        if (col0 == 0)
            for (int i = tid; i < p.dk; i += TILE_THREADS) decays[i] = s_whole;
    }
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const int e = tid + x * TILE_THREADS, col = (e & 31) * 4;
        put_terms<VT>(tv + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), TERM, rv[x].value());
    }
    uint32_t round = 0;
    bool ok = true;
    for (int base = 0; base < p.dk; base += 128, ++round) {
        const int halves = p.dk - base > 64 ? 2 : 1;
        for (int half = 0; half < halves; ++half) {     // 64 channels
            const int i0 = base + half * 64, nk = min(64, p.dk - i0);
            const uint32_t to = tk + half * TILE;
            if (!PER_CHANNEL) {
#pragma unroll
                for (int x = 0; x < NK; ++x) {
                    const int e = tid + x * TILE_THREADS, j = e >> 4;
                    float4 f = rk[x].value();
                    const float w = s_w[j];
                    f.x *= w; f.y *= w; f.z *= w; f.w *= w;
                    put_terms<3>(to + place_in_tile(j, (e & 15) * 4), TERM, f);
                }
            } else {                                    // a thread takes a channel and a quarter of the tokens, from the last back
                constexpr int LEN = CT / 4;
                __shared__ __align__(16) float behind[CT * 64];       // the decays behind a token
                const int i = tid & 63, g = tid >> 6;
                float a[LEN], run = 1.f;
#pragma unroll
                for (int x = 0; x < LEN; ++x) a[x] = g * LEN + x < n && i < nk ? p.dlog[(size_t)(t0 + g * LEN + x) * p.ldd + (size_t)h * p.dk + i0 + i] : 0.f;
#pragma unroll
                for (int x = LEN - 1; x >= 0; --x) {
                    behind[(g * LEN + x) * 64 + i] = run;
                    if (g * LEN + x >= n || i >= nk) continue;
                    const float d = channel_decay<MODE>(a[x], p.decay_scale);
                    run *= d;
                    if (col0 == 0) p.factors[(size_t)(t0 + g * LEN + x) * p.H * p.dk + (size_t)h * p.dk + i0 + i] = d;
                }
                part[g * 64 + i] = run;
                __syncthreads();
#pragma unroll
                for (int x = 0; x < NK; ++x) {
                    const int e = tid + x * TILE_THREADS, j = e >> 4, at = (e & 15) * 4, q = j / LEN;
                    float4 d = *reinterpret_cast<const float4*>(behind + j * 64 + at), f = rk[x].value();
                    for (int later = q + 1; later < 4; ++later) {
                        const float4 more = *reinterpret_cast<const float4*>(part + later * 64 + at);
                        d.x *= more.x; d.y *= more.y; d.z *= more.z; d.w *= more.w;
                    }
                    f.x *= d.x; f.y *= d.y; f.z *= d.z; f.w *= d.w;
                    put_terms<3>(to + place_in_tile(j, at), TERM, f);
                }
                if (tid < nk && col0 == 0) decays[i0 + tid] = (part[tid] * part[64 + tid]) * (part[128 + tid] * part[192 + tid]);
                __syncthreads();
            }
            if (i0 + 64 < p.dk) fetch_k(i0 + 64);
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        const int width = halves * 64;
        if (warp == 0 && elect_one()) {
            tc_fence_after_sync();
            multiply_tiles<VT, 3, true, true>(tmem, tv, TERM, tk, TERM, width);
            mma_commit(&done);
        }
        __syncwarp();
        if (ONES && col0 == 0 && tid < min(width, p.dk - base))         // the column whose values are ones
            added[(size_t)(base + tid) * p.dvp + dvv] = plain_added<TI, MODE>(p, h, base + tid, t0, n, -1, s_w);
        if (ok) ok = wait_done(&done, round & 1, p.status);
        tc_fence_after_sync();
        const int col = (warp & 3) * 32 + lane;
#pragma unroll 1
        for (int at = (warp >> 2) * (width / 2); at < (warp >> 2) * (width / 2) + width / 2; at += 32) {
            float sum[32];
            take_sums<32>(sum, tmem + ((uint32_t)((warp & 3) * 32) << 16) + at, true);
            float* to = added + (size_t)(base + at) * p.dvp + col0 + col;
            if (col < nv) {
                const int rows = min(32, p.dk - base - at);
                uint32_t odd = 0;
#pragma unroll
                for (int x = 0; x < 32; ++x) {
                    odd = max(odd, beyond(sum[x]));
                    if (x < rows) to[(size_t)x * p.dvp] = sum[x];
                }
                if (odd > HELD) mend_added<TI, MODE>(p, to, rows, h, base + at, t0, n, (long long)h * dvv + col0 + col, s_w);
            }
        }
        tc_fence_before_sync();
    }
    leave();
}

// ----------------------------------------------------------------------------- a chunk's outputs, a decay per key channel

// A decay per token and key channel: a block takes the 64 tokens of a chunk and 128 value columns of one head.  The weights P come from
// multiply-adds: pairs of tokens within a block of 16 with their decays as running products (a warp a block and half of the channels), a block's tokens
// against all earlier ones as products of q times the decays since the block's start with k taken on to it (a warp eight channels).  The products with the
// state and with the values run on tcgen05, in three terms per number (one for values that come as bfloat16).
//
// Bound by instruction issue (7,100 per warp when the decays were still taken here from their logits: 103 us for 3,401 tokens of 16 heads of 64 x 128;
// by multiply-adds alone 114): so the first kernel leaves the decays behind.
constexpr int SL = 64;                                  // channels of a slice
// ts, with k, the decays and the warps' sums over it; tq; q; the weights; the blocks' whole decays
constexpr int CHANNEL_SMEM = 1024 + 6 * TILE + 3 * TILE + (SL * CT + CT * PP + 4 * SL) * 4;
static_assert(8 * CROSS * 4 <= 9 * TILE && 2 * SL * CT * 4 <= 6 * TILE, "what lies over the tiles");

// The part of an output that the state gives, by multiply-adds.
template <typename TI, int MODE>
__device__ __noinline__ float plain_from_state(const Scan& p, const float* __restrict__ S, int h, int t0, int t, int col) {
    const TI* q = (const TI*)p.q + (size_t)(t0 + t) * p.ldq + (size_t)(h / p.qk_group) * p.dk;
    float o = 0.f;
    for (int i = 0; i < p.dk && o == o; ++i) {          // NaN stays NaN
        float x = to_f32(q[i]) * (MODE == 1 ? 1.f : p.q_scale);
        for (int j = 0; j < (MODE == 1 ? t : t + 1); ++j) x *= decay_at<MODE>(p, t0 + j, h, i);
        o = fmaf(x, S[(size_t)i * p.dvp + col], o);
    }
    return o;
}

// MANY: more than 128 key channels, more than two runs.
template <typename TI, int MODE, bool MANY>
__global__ void __launch_bounds__(TILE_THREADS, 2)
channel_output_kernel(const __grid_constant__ Scan p) {
    constexpr bool WKV = MODE == 1;
    constexpr int VT = sizeof(TI) == 2 ? 1 : 3, NQ = CT * SL / 4 / TILE_THREADS, NS = 2 * NQ;
    constexpr uint32_t TMEM = 128;                      // two runs' sums [128 columns][64 tokens]
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_slot;
    uint8_t* const base = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    float* const sk = reinterpret_cast<float*>(base);   // [SL][64 tokens]
    float* const sw = sk + SL * CT;                     // the decays [SL][64 tokens]
    float* const sums = sk;                             // [8 warps][CROSS], over k and the decays
    float* const sq = reinterpret_cast<float*>(base + 9 * TILE);         // [SL][64 tokens]
    float* const sp = sq + SL * CT;                     // [64 j][PP]
    float* const edge = sp + CT * PP;                   // [4][SL] the decays of a block of 16 tokens
    const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, half = warp >> 2;
    if (tid == 0) { mbar_init(&done, 1); mbar_fence_init(); }
    if (warp == 0) { tmem_alloc(&tmem_slot, TMEM); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem = tmem_slot, own = tmem + ((uint32_t)(quad * 32) << 16) + half * 32;
    const uint32_t ts = smem_u32(base), tq = ts + 6 * TILE;     // [3][2 halves of the columns][channels], [3][tokens]
    const uint32_t tv = ts, tp = tq;                    // after the slices: [VT][2][tokens], [3][tokens][earlier tokens]
    const int col0 = blockIdx.z * 128, nv = min(128, p.dv - col0);
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.qk_group;
    float* const S = p.chunk_state + ((size_t)c * p.H + h) * p.dk * p.dvp;
    auto leave = [&]() {
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, TMEM);
    };
    if (c == 0)                                         // rows behind the last sequence belong to nobody: a defined value
        for (int t = p.chunk_start[p.n_chunks]; t < p.T_rows; ++t)
            for (int e = tid; e < nv; e += TILE_THREADS) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + col0 + e] = 0.f;
    if (n <= 0 || n > CT) {
        if (n > CT) walk_in_order<TI, MODE>(p, S, c, h, col0, nv, true);
        leave();
        return;
    }
    for (int e = tid; e < CT * PP; e += TILE_THREADS) sp[e] = 0.f;
    const int slices = (p.dk + SL - 1) / SL;
    float out[32];
    bool ok = true;
    for (int s = 0; s < slices; ++s) {
        const int i0 = s * SL, nk = min(SL, p.dk - i0);
        Raw4<TI> rq[NQ], rk[NQ];
        Raw4<float> rd[NQ], rs[NS];
#pragma unroll
        for (int x = 0; x < NQ; ++x) {                  // a warp takes four tokens by 32 channels: no two lanes of a store on one bank
            const int e = tid + x * TILE_THREADS, t = (e >> 6) * 4 + (e >> 3 & 3), i = (e >> 5 & 1) * 32 + (e & 7) * 4;
            get_four(rq[x], (const TI*)p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, t < n, p.vec_q);
            get_four(rk[x], (const TI*)p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, t < n, p.vec_k);
            get_four(rd[x], (const float*)p.factors + (size_t)(t0 + t) * p.H * p.dk + (size_t)h * p.dk + i0, i, nk, t < n, p.vec_d);
        }
        if (s && ok) ok = wait_done(&done, (s - 1) & 1, p.status);
        if (MANY && s >= 2) {
            tc_fence_after_sync();
            take_sums<32>(out, own + (s & 1) * 64, s == 2);
            tc_fence_before_sync();
        }
        if (s) __syncthreads();                         // every warp has seen the products that read what is written over now
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * TILE_THREADS, t = (e >> 6) * 4 + (e >> 3 & 3), i = (e >> 5 & 1) * 32 + (e & 7) * 4;
            const float4 q4 = rq[x].value(), k4 = rk[x].value(), d4 = rd[x].value();
            const float fq[4] = {q4.x, q4.y, q4.z, q4.w}, fk[4] = {k4.x, k4.y, k4.z, k4.w}, fd[4] = {d4.x, d4.y, d4.z, d4.w};
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                const int at = at_ct(i + y, t);
                sq[at] = WKV ? fq[y] : fq[y] * p.q_scale;
                sk[at] = fk[y];
                sw[at] = t < n && i + y < nk ? fd[y] : 1.f;
            }
        }
        // the state's slice on its way to registers
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * TILE_THREADS, i = e >> 5;
            get_four(rs[x], S + (size_t)(i0 + i) * p.dvp, col0 + (e & 31) * 4, (p.dv + 3) / 4 * 4, i < nk, 1);
        }
        __syncthreads();
        // pairs of tokens within a block of 16: lane = token j and a quarter of the channels
        {
            const int jj = lane & 15, b0 = quad * 16, e0 = (half * 2 + (lane >> 4)) * (SL / 4);
            float d[16];
#pragma unroll
            for (int x = 0; x < 16; ++x) d[x] = 0.f;
            for (int i = e0; i < e0 + SL / 4; ++i) {
                float fq[16], fw[16];
#pragma unroll
                for (int g = 0; g < 4; ++g) {
                    const float4 x = *reinterpret_cast<const float4*>(sq + at_ct(i, b0 + 4 * g)), y = *reinterpret_cast<const float4*>(sw + at_ct(i, b0 + 4 * g));
                    fq[4 * g] = x.x; fq[4 * g + 1] = x.y; fq[4 * g + 2] = x.z; fq[4 * g + 3] = x.w;
                    fw[4 * g] = y.x; fw[4 * g + 1] = y.y; fw[4 * g + 2] = y.z; fw[4 * g + 3] = y.w;
                }
                const float kj = sk[at_ct(i, b0 + jj)];
                const float u = WKV && i < nk ? load_as_f32(p.bonus, p.bonus_dtype, (size_t)h * p.dk + i0 + i) : 1.f;
                float run = kj;
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    if (x > jj && !WKV) run *= fw[x];
                    d[x] = fmaf(fq[x], WKV && x == jj ? u * kj : run, d[x]);         // means nothing where x < jj
                    if (x > jj && WKV) run *= fw[x];
                }
            }
#pragma unroll
            for (int x = 0; x < 16; ++x) d[x] += __shfl_xor_sync(0xffffffffu, d[x], 16);
#pragma unroll
            for (int turn = 0; turn < 2; ++turn) {      // the channels' halves one after the other
                if (half == turn && lane < 16)
#pragma unroll
                    for (int x = 0; x < 16; ++x) if (x >= jj) sp[(b0 + jj) * PP + b0 + x] += d[x];
                __syncthreads();
            }
        }
        // q times the decays since the start of its block of 16, k times those up to the block's end, the block's whole decay
        {
            const int i = (tid & 15) * 4 + (tid >> 4 & 3), g = tid >> 6;       // neighbouring lanes four channels apart: other banks
            float4 w[4];
            float run = 1.f;
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                w[x] = *reinterpret_cast<const float4*>(sw + at_ct(i, g * 16 + 4 * x));
                float4* at = reinterpret_cast<float4*>(sq + at_ct(i, g * 16 + 4 * x));
                float4 f = *at;
                if (!WKV) run *= w[x].x;
                f.x *= run; run *= WKV ? w[x].x : w[x].y;
                f.y *= run; run *= WKV ? w[x].y : w[x].z;
                f.z *= run; run *= WKV ? w[x].z : w[x].w;
                f.w *= run;
                if (WKV) run *= w[x].w;
                *at = f;
            }
            edge[g * SL + i] = run;
            run = 1.f;
#pragma unroll
            for (int x = 3; x >= 0; --x) {
                float4* at = reinterpret_cast<float4*>(sk + at_ct(i, g * 16 + 4 * x));
                float4 f = *at;
                f.w *= run; run *= w[x].w;
                f.z *= run; run *= w[x].z;
                f.y *= run; run *= w[x].y;
                f.x *= run; run *= w[x].x;
                *at = f;
            }
        }
        __syncthreads();
        // a block's tokens against all earlier ones, whose k are taken on to this block's start; a warp has eight of the channels
        f32x2 x1[2][2], x2[4][2], x3[6][2];
#pragma unroll
        for (int x = 0; x < 6; ++x) {
            if (x < 2) x1[x][0] = x1[x][1] = 0ull;
            if (x < 4) x2[x][0] = x2[x][1] = 0ull;
            x3[x][0] = x3[x][1] = 0ull;
        }
        const int ch = warp * 8 + (lane & 7), piece = (lane >> 3) * 4;
        cross_product<1, 8, at_ct>(x1, sq, sk, warp * 8, lane);
        __syncwarp();
        scale_four(sk + at_ct(ch, piece), edge[SL + ch]);
        __syncwarp();
        cross_product<2, 8, at_ct>(x2, sq, sk, warp * 8, lane);
        __syncwarp();
        scale_four(sk + at_ct(ch, piece), edge[2 * SL + ch]);
        scale_four(sk + at_ct(ch, 16 + piece), edge[2 * SL + ch]);
        __syncwarp();
        cross_product<3, 8, at_ct>(x3, sq, sk, warp * 8, lane);
        __syncthreads();
        // the warps' sums over k and the decays, then added up
        cross_store<1>(sums + warp * CROSS, x1, lane);
        cross_store<2>(sums + warp * CROSS, x2, lane);
        cross_store<3>(sums + warp * CROSS, x3, lane);
        __syncthreads();
#pragma unroll
        for (int pair = 0; pair < 6; ++pair) {          // blocks (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
            const int I = pair == 0 ? 1 : pair < 3 ? 2 : 3, J = pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3;
            const int t = tid & 15, j = J * 16 + (tid >> 4);
            const float* at = sums + cross_at(I) + t * (16 * I + 1) + j;
            float sum = 0.f;
#pragma unroll
            for (int w = 0; w < 8; w += 2) sum += at[w * CROSS] + at[(w + 1) * CROSS];
            sp[j * PP + I * 16 + t] += sum;
        }
        __syncthreads();
        // the state, and q times the decays since the chunk's start, as terms
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * TILE_THREADS, col = (e & 31) * 4;
            put_terms<3>(ts + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, rs[x].value());
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {                   // a thread takes a token's eight channels, lanes neighbouring tokens
            const int e = tid + x * TILE_THREADS, t = e & 63, i = (e >> 6) * 8;
            float f[8];
#pragma unroll
            for (int y = 0; y < 8; ++y) {
                float before = 1.f;
                for (int m = 0; m < t / 16; ++m) before *= edge[m * SL + i + y];
                f[y] = sq[at_ct(i + y, t)] * before;
            }
            put_eight(tq + place_in_tile(t, i), TILE, f);
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after_sync();
            multiply_tiles<3, 3, true, false>(tmem + (s & 1) * 64, ts, 2 * TILE, tq, TILE, CT);       // S0^T q
            mma_commit(&done);
        }
        __syncwarp();
    }
    Raw4<TI> rv[NS];
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * TILE_THREADS, j = e >> 5;
        get_four(rv[x], (const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)h * p.dv + col0, (e & 31) * 4, nv, j < n, p.vec_v);
    }
    if (ok) ok = wait_done(&done, (slices - 1) & 1, p.status);
    tc_fence_after_sync();
    const int older = slices & 1, newer = older ^ 1;
    if (slices > 1) take_sums<32>(out, own + older * 64, slices == 2);
    take_sums<32>(out, own + newer * 64, slices == 1);
    tc_fence_before_sync();
    __syncthreads();                                    // every warp has seen the products: their tiles may be written over
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * TILE_THREADS, col = (e & 31) * 4;
        put_terms<VT>(tv + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, rv[x].value());
    }
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int e = tid + x * TILE_THREADS, t = e & 63, j = (e >> 6) * 8;
        float f[8];
#pragma unroll
        for (int y = 0; y < 8; ++y) f[y] = sp[(j + y) * PP + t];
        put_eight(tp + place_in_tile(t, j), TILE, f);
    }
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0 && elect_one()) {
        tc_fence_after_sync();
        multiply_tiles<VT, 3, true, false>(tmem, tv, 2 * TILE, tp, TILE, CT);       // V^T P^T
        mma_commit(&done);
    }
    __syncwarp();
    if (ok) ok = wait_done(&done, slices & 1, p.status);
    tc_fence_after_sync();
    float more[32];
    take_sums<32>(more, own, true);
    const int in = quad * 32 + lane, rows = n - half * 32;
    if (in < nv) {
        float* const o = p.o + (size_t)t0 * p.ldo + (size_t)h * p.dv + col0 + in;
        uint32_t odd = 0;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            odd = max(odd, beyond(out[x] + more[x]));
            if (x < rows) o[(size_t)(half * 32 + x) * p.ldo] = out[x] + more[x];
        }
        if (odd > HELD)                                 // by multiply-adds, where the terms did not hold the operands: a later token's value meets no earlier one
            for (int t = half * 32; t < min(n, half * 32 + 32); ++t) {
                if (held(o[(size_t)t * p.ldo])) continue;
                float v = plain_from_state<TI, MODE>(p, S, h, t0, t, col0 + in);
                for (int j = 0; j <= t && v == v; ++j)
                    v = fmaf(sp[j * PP + t], to_f32(((const TI*)p.v)[(size_t)(t0 + j) * p.ldv + (size_t)h * p.dv + col0 + in]), v);
                o[(size_t)t * p.ldo] = v;
            }
    }
    leave();
}

// ----------------------------------------------------------------------------- a chunk's outputs, one decay per head

// A block takes the 64 tokens of a chunk and 128 value columns of one head, or (NH = 2) 64 of each of two neighbouring heads that share
// q and k, whose products q k^T are then taken once.  The key channels pass in slices of 64 through shared memory, as terms: q, k and v in QT
// (one where they come as bfloat16), the states and the weights in three.  A slice is a run in the tensor unit; the runs' sums, from two sets
// of accumulators, are added in registers.  Columns on the TMEM lanes for the outputs, tokens for q k^T.
template <typename TI, int NH> constexpr int tile_smem() {
    const int qt = sizeof(TI) == 2 ? 1 : 3, slices = (2 * qt + 6) * TILE, weights = (3 * NH + 2 * qt) * TILE;
    return 1024 + (slices > weights ? slices : weights);
}

// One output by multiply-adds, where the terms did not hold what went into it.  The weights are taken from their terms at `tp` where these held them.
template <typename TI, int MODE>
__device__ __noinline__ float plain_output(const Scan& p, const float* __restrict__ S, const float* __restrict__ a, const float* __restrict__ b, float cum,
                                           uint32_t tp, int h, int t0, int t, int col) {
    constexpr bool ONES = MODE == 2;
    const int hq = h / p.qk_group, dvv = ONES ? p.dv - 1 : p.dv;
    const TI* q = (const TI*)p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk;
    float o = 0.f, d = 1.f;
    for (int i = 0; i < p.dk; ++i) o = fmaf(to_f32(q[i]) * p.q_scale, S[(size_t)i * p.dvp + col], o);
    o *= cum;
    for (int j = t; j >= 0 && o == o; --j) {           // NaN stays NaN
        float w = 0.f;
        for (int i = 2; i >= 0; --i) {
            uint16_t term;
            asm volatile("ld.shared.u16 %0, [%1];" : "=h"(term) : "r"(tp + i * TILE + place_in_tile(t, j)));
            w += __uint_as_float((uint32_t)term << 16);
        }
        if (!held(w)) {
            const TI* k = (const TI*)p.k + (size_t)(t0 + j) * p.ldk + hq * p.dk;
            float raw = 0.f;
            for (int i = 0; i < p.dk; ++i) raw = fmaf(to_f32(q[i]) * p.q_scale, to_f32(k[i]), raw);
            w = b[j] * d * raw;
        }
        o = fmaf(w, ONES && col == dvv ? 1.f : to_f32(((const TI*)p.v)[(size_t)(t0 + j) * p.ldv + (size_t)h * dvv + col]), o);
        d = times_decay<MODE>(d, a[j]);
    }
    return o;
}

// MANY: more than 128 key channels, more than two runs; without it no sums are held while slices pass.
template <typename TI, int MODE, int NH, bool MANY>
__global__ void __launch_bounds__(TILE_THREADS, 2)
tile_output_kernel(const __grid_constant__ Scan p) {
    constexpr bool ONES = MODE == 2;
    constexpr int QT = sizeof(TI) == 2 ? 1 : 3, NQ = CT * 16 / TILE_THREADS, NS = 2 * NQ;
    constexpr uint32_t TMEM = 256;                      // two runs' sums: the outputs [128 columns][64 tokens], q k^T [64 tokens (128 lanes)][64]
    extern __shared__ uint8_t smem_raw[];
    __shared__ float s_a[NH][CT], s_cum[NH][CT], s_b[NH][CT], s_ones[2][CT];
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_slot;
    const int c = blockIdx.x, h = blockIdx.y * NH, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, half = warp >> 2;
    if (tid == 0) { mbar_init(&done, 1); mbar_fence_init(); }
    if (warp == 0) { tmem_alloc(&tmem_slot, TMEM); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem = tmem_slot, own = tmem + ((uint32_t)(quad * 32) << 16) + half * 32;
    const uint32_t tq = (smem_u32(smem_raw) + 1023) & ~1023u, tk = tq + QT * TILE, ts = tk + QT * TILE;     // [QT][tokens], [QT][tokens], [3][2 halves of the columns][channels]
    const uint32_t tp = tq, tv = tp + 3 * NH * TILE;    // after the slices: [NH][3][tokens][earlier tokens], [QT][2][tokens]
    const int dvv = ONES ? p.dv - 1 : p.dv, col0 = blockIdx.z * 128, nv = NH == 2 ? dvv : min(128, dvv - col0);
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.qk_group;
    auto leave = [&]() {
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, TMEM);
    };
    if (c == 0)                                         // rows behind the last sequence belong to nobody: a defined value
        for (int t = p.chunk_start[p.n_chunks]; t < p.T_rows; ++t) {
            for (int e = tid; e < NH * nv; e += TILE_THREADS) p.o[(size_t)t * p.ldo + (size_t)(h + e / nv) * p.dv + (NH == 2 ? 0 : col0) + e % nv] = 0.f;
            if (ONES && col0 == 0 && tid == 0) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + dvv] = 0.f;
        }
    if (n <= 0 || n > CT) {
        if (n > CT)
            for (int x = 0; x < NH; ++x) {
                float* S = p.chunk_state + ((size_t)c * p.H + h + x) * p.dk * p.dvp;
                walk_in_order<TI, MODE>(p, S, c, h + x, col0, nv, true);
                if (ONES && col0 == 0) walk_in_order<TI, MODE>(p, S, c, h + x, dvv, 1, true);
            }
        leave();
        return;
    }
    for (int e = tid; e < NH * CT; e += TILE_THREADS) { // the tokens' decays and weights
        const int x = e / CT, t = e % CT;
        s_a[x][t] = t < n ? decay_at<MODE>(p, t0 + t, h + x, 0) : (MODE == 5 ? 0.f : 1.f);
        s_b[x][t] = t >= n ? 0.f : (MODE == 2 || MODE == 5) ? p.gb[(size_t)(t0 + t) * p.ldg + h + x] : 1.f;
    }
    float out[32], raw[32], ones_part = 0.f;            // column quad 32 + lane of tokens half 32 ..; token quad 32 + lane (< 64) against tokens half 32 ..
    const int slices = (p.dk + 63) / 64;
    bool ok = true;
    for (int s = 0; s < slices; ++s) {
        const int i0 = s * 64, nk = min(64, p.dk - i0);
        Raw4<float> rs[NS];
        Raw4<TI> rq[NQ], rk[NQ];
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * TILE_THREADS, t = e >> 4, i = (e & 15) * 4;
            get_four(rq[x], (const TI*)p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, t < n, p.vec_q);
            get_four(rk[x], (const TI*)p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, t < n, p.vec_k);
        }
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * TILE_THREADS, i = e >> 5, col = (e & 31) * 4, at = NH == 2 ? col & 63 : col0 + col;
            get_four(rs[x], p.chunk_state + (((size_t)c * p.H + h + (NH == 2 ? col >> 6 : 0)) * p.dk + i0 + i) * p.dvp, at, (dvv + 3) / 4 * 4, i < nk, 1);
        }
        if (s && ok) ok = wait_done(&done, (s - 1) & 1, p.status);
        if (MANY && s >= 2) {                                 // the set of accumulators that comes next is full: onto the thread's sums
            tc_fence_after_sync();
            take_sums<32>(out, own + (s & 1) * 128, s == 2);
            if (quad < 2) take_sums<32>(raw, own + (s & 1) * 128 + 64, s == 2);
        }
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * TILE_THREADS;
            const uint32_t at = place_in_tile(e >> 4, (e & 15) * 4);
            put_terms<QT>(tq + at, TILE, rq[x].value());
            put_terms<QT>(tk + at, TILE, rk[x].value());
        }
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * TILE_THREADS, col = (e & 31) * 4;
            put_terms<3>(ts + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, rs[x].value());
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after_sync();
            multiply_tiles<3, QT, true, false>(tmem + (s & 1) * 128, ts, 2 * TILE, tq, TILE, CT);           // S0^T q
            multiply_tiles<QT, QT, false, false>(tmem + (s & 1) * 128 + 64, tq, TILE, tk, TILE, CT);        // q k^T
            mma_commit(&done);
        }
        __syncwarp();
        if (s == 0)
            for (int e = tid; e < NH * CT; e += TILE_THREADS) {         // the decays since the chunk's start
                const int x = e / CT, t = e % CT;
                float cum = 1.f;
                if constexpr (MODE == 0) cum = decay_power(s_a[x][0], min(t + 1, n));
                else
#pragma unroll 8
                    for (int j = 0; j < CT; ++j) if (j <= t) cum = times_decay<MODE>(cum, s_a[x][j]);
                s_cum[x][t] = cum;
            }
        if (ONES && blockIdx.z == 0 && tid < n) {
            const float* last = p.chunk_state + (((size_t)c * p.H + h) * p.dk + i0) * p.dvp + dvv;
            const TI* q = (const TI*)p.q + (size_t)(t0 + tid) * p.ldq + hq * p.dk + i0;
            for (int i = 0; i < nk; ++i) ones_part = fmaf(to_f32(q[i]), last[(size_t)i * p.dvp], ones_part);
        }
    }
    Raw4<TI> rv[NS];
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * TILE_THREADS, j = e >> 5, col = (e & 31) * 4, head = NH == 2 ? col >> 6 : 0, at = NH == 2 ? col & 63 : col;
        get_four(rv[x], (const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)(h + head) * dvv + (NH == 2 ? 0 : col0), at, nv, j < n, p.vec_v);
    }
    if (ok) ok = wait_done(&done, (slices - 1) & 1, p.status);
    tc_fence_after_sync();
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * TILE_THREADS, col = (e & 31) * 4;
        put_terms<QT>(tv + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, rv[x].value());
    }
    const int older = slices & 1, newer = older ^ 1;    // the sets of the last run but one and of the last
    if (quad < 2) {                                     // the weights P[t][j]: a thread half of a token's, from the last earlier token back
        if (slices > 1) take_sums<32>(raw, own + older * 128 + 64, slices == 2);
        take_sums<32>(raw, own + newer * 128 + 64, slices == 1);
        const int t = quad * 32 + lane;
#pragma unroll
        for (int x = 0; x < NH; ++x) {
            float d = 1.f, ones = 0.f;
            if (half == 0)
#pragma unroll 8
                for (int j = CT - 2; j >= 32; --j) if (j < t) d = times_decay<MODE>(d, s_a[x][j + 1]);
#pragma unroll
            for (int j8 = 24; j8 >= 0; j8 -= 8) {
                float w[8];
#pragma unroll
                for (int y = 7; y >= 0; --y) {
                    const int j = half * 32 + j8 + y;
                    if (j < t) d = times_decay<MODE>(d, s_a[x][j + 1]);
                    // a weight of zero stays zero whatever the product is: a token's q never meets a later token's k
                    w[y] = j <= t ? s_b[x][j] * d * (raw[j8 + y] * p.q_scale) : 0.f;
                    if (ONES) ones += w[y];
                }
                put_eight(tp + x * 3 * TILE + place_in_tile(t, half * 32 + j8), TILE, w);
            }
            if (ONES) s_ones[half][t] = ones;
        }
    }
    if (slices > 1) take_sums<32>(out, own + older * 128, slices == 2);
    take_sums<32>(out, own + newer * 128, slices == 1);
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0 && elect_one()) {
        tc_fence_after_sync();
#pragma unroll
        for (int x = 0; x < NH; ++x) multiply_tiles<QT, 3, true, false>(tmem + x * 64, tv, 2 * TILE, tp + x * 3 * TILE, TILE, CT);       // V^T P^T
        mma_commit(&done);
    }
    __syncwarp();
    const int head = NH == 2 ? quad >> 1 : 0, in = quad * 32 + lane, col = NH == 2 ? in & 63 : col0 + in;
    const float* const S = p.chunk_state + ((size_t)c * p.H + h + head) * p.dk * p.dvp;
#pragma unroll
    for (int x = 0; x < 32; ++x) out[x] *= s_cum[head][half * 32 + x] * p.q_scale;
    if (ONES && blockIdx.z == 0 && tid < n) {
        float sum = fmaf(s_cum[0][tid] * p.q_scale, ones_part, s_ones[0][tid] + s_ones[1][tid]);
        if (!held(sum)) sum = plain_output<TI, MODE>(p, S, s_a[0], s_b[0], s_cum[0][tid], tp, h, t0, tid, dvv);
        p.o[(size_t)(t0 + tid) * p.ldo + (size_t)h * p.dv + dvv] = sum;
    }
    if (ok) ok = wait_done(&done, slices & 1, p.status);
    tc_fence_after_sync();
    take_sums<32>(out, own + head * 64, false);
    float* const o = p.o + (size_t)t0 * p.ldo + (size_t)(h + head) * p.dv + col;
    if (col < dvv) {
        const int rows = n - half * 32;
        uint32_t odd = 0;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            odd = max(odd, beyond(out[x]));
            if (x < rows) o[(size_t)(half * 32 + x) * p.ldo] = out[x];
        }
        if (odd > HELD)
            for (int t = half * 32; t < min(n, half * 32 + 32); ++t)
                if (!held(o[(size_t)t * p.ldo])) o[(size_t)t * p.ldo] = plain_output<TI, MODE>(p, S, s_a[head], s_b[head], s_cum[head][t], tp + head * 3 * TILE, h + head, t0, t, col);
    }
    leave();
}

template <typename TI, int MODE>
int launch_added(const Scan& p, int n_chunks, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv, smem = added_smem<TI>();
    cudaError_t e = cudaFuncSetAttribute(added_state_kernel<TI, MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e == cudaSuccess)
        e = qs_launch_dependent(added_state_kernel<TI, MODE>, dim3(n_chunks, p.H, (dvv + 127) / 128), dim3(TILE_THREADS), smem, stream, p);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "state_scan, added states: %s", cudaGetErrorString(e));
    return qs_check_launch("state_scan, added states");
}

template <typename TI, int MODE, int NH>
int launch_output(const Scan& p, int n_chunks, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    const dim3 grid(n_chunks, p.H / NH, NH == 2 ? 1 : (dvv + 127) / 128);
    cudaError_t e;
    if constexpr (MODE == 1 || MODE == 4) {
        const auto kernel = p.dk > 128 ? channel_output_kernel<TI, MODE, true> : channel_output_kernel<TI, MODE, false>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, CHANNEL_SMEM);
        if (e == cudaSuccess) e = qs_launch_dependent(kernel, grid, dim3(TILE_THREADS), CHANNEL_SMEM, stream, p);
    } else {
        constexpr int smem = tile_smem<TI, NH>();
        const auto kernel = p.dk > 128 ? tile_output_kernel<TI, MODE, NH, true> : tile_output_kernel<TI, MODE, NH, false>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess) e = qs_launch_dependent(kernel, grid, dim3(TILE_THREADS), smem, stream, p);
    }
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "state_scan, chunk outputs: %s", cudaGetErrorString(e));
    return qs_check_launch("state_scan, chunk outputs");
}

template <typename TI, int MODE>
int run(const Scan& p, int n_chunks, bool outputs, cudaStream_t stream) {
    if (!outputs) return launch_added<TI, MODE>(p, n_chunks, stream);
    if constexpr (MODE == 5)                            // two heads that share q and k: their products once
        if (p.dv <= 64 && p.qk_group % 2 == 0) return launch_output<TI, MODE, 2>(p, n_chunks, stream);
    return launch_output<TI, MODE, 1>(p, n_chunks, stream);
}

template <typename TI>
int pick(int mode, const Scan& p, int n_chunks, bool outputs, cudaStream_t stream) {
    switch (mode) {
        case 0: return run<TI, 0>(p, n_chunks, outputs, stream);
        case 1: return run<TI, 1>(p, n_chunks, outputs, stream);
        case 2: return run<TI, 2>(p, n_chunks, outputs, stream);
        case 4: return run<TI, 4>(p, n_chunks, outputs, stream);
        case 5: return run<TI, 5>(p, n_chunks, outputs, stream);
    }
    return qs_fail(QS_ERR_INVALID_INPUT, "state_scan: mode %d has no chunks", mode);
}

// The activation of q, k and v, once per element, for chunks whose kernels read them several times.
template <typename TI>
__global__ void __launch_bounds__(256)
activate_rows_kernel(float* __restrict__ out, const TI* __restrict__ q, size_t ldq, const TI* __restrict__ k, size_t ldk, const TI* __restrict__ v, size_t ldv,
                     int nk, int nv, int act) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t t = blockIdx.x;
    const int n = 2 * nk + nv;
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const TI* src = i < nk ? q + t * ldq + i : i < 2 * nk ? k + t * ldk + i - nk : v + t * ldv + i - 2 * nk;
        out[t * n + i] = apply_activation(to_f32(*src), act);
    }
}
template <typename TI>
__global__ void __launch_bounds__(256)
activate_fours_kernel(float4* __restrict__ out, const TI* __restrict__ q, size_t ldq, const TI* __restrict__ k, size_t ldk, const TI* __restrict__ v, size_t ldv,
                      int nk4, int nv4, int act) {
    grid_dep_launch();
    grid_dep_wait();
    const size_t t = blockIdx.x;
    const int n = 2 * nk4 + nv4;
    for (int i = threadIdx.x + blockIdx.y * blockDim.x; i < n; i += blockDim.x * gridDim.y) {
        const TI* src = i < nk4 ? q + t * ldq + 4 * i : i < 2 * nk4 ? k + t * ldk + 4 * (i - nk4) : v + t * ldv + 4 * (i - 2 * nk4);
        Raw4<TI> r;
        r.get(src);
        float4 f = r.value();
        f.x = apply_activation(f.x, act); f.y = apply_activation(f.y, act); f.z = apply_activation(f.z, act); f.w = apply_activation(f.w, act);
        out[t * n + i] = f;
    }
}

}  // namespace

// out [rows][2 nk + nv] = act(q), act(k), act(v) side by side, in 32-bit.
QS_API int qs_scan_activate(float* out, const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv, int dtype, int rows, int nk, int nv,
                            int act, cudaStream_t stream) {
    if (rows == 0) return QS_OK;
    QS_REQUIRE(rows > 0 && nk > 0 && nv > 0 && (dtype == QS_F32 || dtype == QS_BF16), "scan_activate: bad sizes");
    const size_t item = dtype == QS_F32 ? 4 : 2;
    auto fits = [&](const void* ptr, long long ld) { return ld % 4 == 0 && ((uintptr_t)ptr % (4 * item)) == 0; };
    const bool fours = nk % 4 == 0 && nv % 4 == 0 && fits(q, ldq) && fits(k, ldk) && fits(v, ldv);
    cudaError_t e;
#define GO(T) do { if (fours) e = qs_launch_dependent(activate_fours_kernel<T>, dim3(rows, 2), dim3(256), 0, stream, (float4*)out, (const T*)q, (size_t)ldq, \
        (const T*)k, (size_t)ldk, (const T*)v, (size_t)ldv, nk / 4, nv / 4, act); \
    else e = qs_launch_dependent(activate_rows_kernel<T>, dim3(rows), dim3(256), 0, stream, out, (const T*)q, (size_t)ldq, (const T*)k, (size_t)ldk, (const T*)v, \
        (size_t)ldv, nk, nv, act); } while (0)
    if (dtype == QS_F32) GO(float); else GO(__nv_bfloat16);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "scan_activate: %s", cudaGetErrorString(e));
    return qs_check_launch("scan_activate");
}

// The first (outputs == 0: chunk_state becomes what every chunk adds, chunk_decay its decays) and the last kernel (chunk_state
// holds the states the chunks start from) of a scan in chunks; operands as for `qs_state_scan`.
int qs_scan_chunks(int mode, int outputs, float* o, long long ldo, const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                   int dtype, const float* dlog, long long ldd, const float* head_decay, const void* bonus, int bonus_dtype, int H, int dk, int dv,
                   const int32_t* chunk_start, int n_chunks, int T_rows, float* chunk_state, float* chunk_decay, const float* ga, const float* gb,
                   long long ldg, float q_scale, int qk_group, float decay_scale, float* chunk_factors, int32_t* status, cudaStream_t stream) {
    const size_t item = dtype == QS_F32 ? 4 : 2;
    auto fours = [&](const void* ptr, long long ld, int per_head) { return (int)(per_head % 4 == 0 && ld % 4 == 0 && ((uintptr_t)ptr % (4 * item)) == 0); };
    Scan p = {};
    p.q = q; p.k = k; p.v = v; p.ldq = (size_t)ldq; p.ldk = (size_t)ldk; p.ldv = (size_t)ldv;
    p.dlog = dlog; p.ldd = (size_t)ldd; p.head_decay = head_decay; p.ga = ga; p.gb = gb; p.ldg = (size_t)ldg;
    p.bonus = bonus; p.bonus_dtype = bonus_dtype; p.chunk_start = chunk_start; p.chunk_state = chunk_state; p.chunk_decay = chunk_decay;
    p.o = o; p.ldo = (size_t)ldo; p.H = H; p.dk = dk; p.dv = dv; p.dvp = (dv + 3) / 4 * 4; p.qk_group = qk_group;
    p.q_scale = q_scale; p.decay_scale = decay_scale;
    p.vec_q = fours(q, ldq, dk); p.vec_k = fours(k, ldk, dk); p.vec_v = fours(v, ldv, mode == 2 ? dv - 1 : dv);
    p.factors = chunk_factors;
    p.vec_d = dk % 4 == 0 && ((uintptr_t)chunk_factors % 16) == 0;
    p.n_chunks = n_chunks; p.T_rows = T_rows; p.status = status;
    return dtype == QS_F32 ? pick<float>(mode, p, n_chunks, outputs != 0, stream) : pick<__nv_bfloat16>(mode, p, n_chunks, outputs != 0, stream);
}
