// The matrix-state recurrences of recurrent.cu over long prompts: chunks of up to 64 tokens as matrix products.
//
// Within a chunk that starts from the state S0 (a column of S per value dim, channels i of the keys)
//       o_t = (q_t * cum_t)^T S0 + sum_{j <= t} P[t][j] v_j,      P[t][j] = b_j sum_i q_t[i] k_j[i] (a_{j+1} .. a_t)[i],
//       S_end = diag(a_1 .. a_n) S0 + sum_j b_j (a_{j+1} .. a_n * k_j) v_j^T,        cum_t = a_1 .. a_t,
// with a the decays (one number per token and head, or one per token and key channel) and b the input weights.  Three kernels
// take a prompt's chunks side by side:
//   added_state_kernel      what each chunk adds to the state it starts from, and its decays
//   chunk_prefix_kernel     (recurrent.cu) the state each chunk starts from, and the sequence's last one
//   chunk_output_kernel     every token's o, written once
// Decays enter as products of at most 64 factors up to one, never as quotients, so small ones cost no precision: per token and head by a
// recursion from a token back over the earlier ones; per channel in blocks of 16 tokens, a block's own pairs walked in order, pairs of blocks
// through the products up to the blocks' common edge.
//
// The products of 32-bit numbers run on tcgen05 as products of bfloat16 terms (terms.cuh), in runs of 64 whose sums are added outside; against
// float64 they are nearer than the multiply-adds that stood here before (o, 2-norm: state-space form 1.4e-7 instead of 1.5e-7, gated memory
// 1.4e-7 instead of 1.9e-7, decay per head 7.9e-7 instead of 8.8e-7).  q, k and v that come as bfloat16 are one term: q k^T is then one product instead
// of six.  Bound by each block's chain of fetch, split, barrier, MMAs and stores at two blocks per SM (leaving out the MMAs: 63 of 76 us
// for the outputs, 42 of 47 for what the chunks add, at 4,096 tokens of 16 heads of 128 x 128, float32 operands); the split needs half of
// the issue slots.  On mma.sync the same products took 138 and 59 us, multiply-adds 139 and 66.
//
// Microseconds of the scan alone (multiply-adds | now; caches flushed): decay per head, 4,096 tokens, 16 heads of 128 x 128, float32: 236 | 151; 1,000
// tokens, bfloat16: 85 | 38; state-space form, 2,048 tokens, 64 heads of 128 x 64: 237 | 142; gated memory, 1,000 tokens, 4 heads of 256 x 256:
// 136 | 79; per channel (its outputs on the CUDA cores), 3,401 tokens, 16 heads of 64 x 128: 175 | 163.
#include "scan.cuh"
#include "scan_tiles.cuh"
#include "term_tiles.cuh"

namespace {

struct Scan {
    const void *q, *k, *v;
    size_t ldq, ldk, ldv;
    const float *dlog; size_t ldd;                      // per channel: logits of the decays
    const float *head_decay;                            // one decay per head
    const float *ga, *gb; size_t ldg;                   // per token and head: decays (less one in mode 5), input weights
    const void* bonus; int bonus_dtype;
    const int32_t* chunk_start;
    float *chunk_state, *chunk_decay;                   // [chunks][H][dk][dvp], [chunks][H][dk]
    float* o; size_t ldo;
    int H, dk, dv, dvp, qk_group, n_chunks, T_rows;       // dvp: dv rounded up to a multiple of four
    float q_scale, decay_scale;
    int vec_q, vec_k, vec_v, vec_o;                    // whether rows may be read (written) in pieces of four
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

// A block takes 64 NC value columns of one head's state, up to 128 key channels at a time: added[i][col] = sum_j kw_j[i] v_j[col], the
// tokens on the sum's side, kw_j = b_j k_j times the decays behind token j.  kw in three terms, v in VT (one where it comes as bfloat16).
// Columns on the TMEM lanes, so that a warp writes 32 neighbouring ones.
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
// The sums of a column that the terms gave no number for.
template <typename TI, int MODE>
__device__ __noinline__ void mend_added(const Scan& p, float* to, int rows, int h, int i, int t0, int n, long long v_at, const float* s_w) {
    for (int x = 0; x < rows; ++x)
        if (!is_number(to[(size_t)x * p.dvp])) to[(size_t)x * p.dvp] = plain_added<TI, MODE>(p, h, i + x, t0, n, v_at, s_w);
}

template <typename TI> constexpr int added_smem() { return 1024 + (3 + (sizeof(TI) == 2 ? 1 : 3)) * 2 * TILE; }

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
#pragma unroll 8
            for (int t = CT - 1; t > 0; --t) if (t > tid) w = times_decay<MODE>(w, s_a[t]);
            if (tid == 0) s_whole = times_decay<MODE>(w, s_a[0]);
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
                    run *= g * LEN + x < n && i < nk ? channel_decay<MODE>(a[x], p.decay_scale) : 1.f;
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
                bool odd = false;
#pragma unroll
                for (int x = 0; x < 32; ++x) {
                    odd |= !is_number(sum[x]);
                    if (x < rows) to[(size_t)x * p.dvp] = sum[x];
                }
                if (odd) mend_added<TI, MODE>(p, to, rows, h, base + at, t0, n, (long long)h * dvv + col0 + col, s_w);
            }
        }
        tc_fence_before_sync();
    }
    leave();
}

// ----------------------------------------------------------------------------- a chunk's outputs

// A block takes the 64 tokens of a chunk and 64 NC value columns: of one head, or (NH = 2) 64 of each of two neighbouring heads
// that share q and k, whose products q k^T are then taken once.  The key channels pass in slices through shared memory.
// Three blocks per SM leave a thread 168 registers.  The bfloat16 forms fit (at most 16 bytes spilled); the float32 ones, which a decay per head
// behind an activation takes too, hold a slice of q and k on its way in twice the room and spill 340 bytes, 700 to 780 per channel and with
// the column of ones.
template <int MODE, int NC>
constexpr int output_body() {                           // floats of shared memory before the weights
    const int sl = MODE == 1 || MODE == 4 ? 64 : 32, stage = sl == 64 ? (3 * sl * CT > sl * CT + sl * 64 * NC ? 3 * sl * CT : sl * CT + sl * 64 * NC)
                                                                      : 2 * sl * CT + 2 * sl * 64 * NC;
    return stage > CT * 64 * NC ? stage : CT * 64 * NC;
}

template <typename TI, int MODE, int NC, int NH>
__global__ void __launch_bounds__(THREADS, 3)
chunk_output_kernel(Scan p) {
    constexpr bool PER_CHANNEL = MODE == 1 || MODE == 4, ONES = MODE == 2, WKV = MODE == 1;
    constexpr int SL = PER_CHANNEL ? 64 : 32;           // channels of a slice
    constexpr int COLS = 64 * NC, NQ = CT * SL / 4 / THREADS, NV = CT * 16 * NC / THREADS;
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                                   // [SL][64 tokens]
    float* sk = sq + SL * CT;                           // [SL][64 tokens]
    float* sw = sk + SL * CT;                           // PER_CHANNEL: the decays [SL][64 tokens]; then the state lies over sk, sw
    float* ss = PER_CHANNEL ? sk : sw;                  // [SL][COLS]: a slice of the states the chunk starts from; two of them in turn per head
    float* svv = smem;                                  // [64 tokens][COLS]: the values, after the last slice
    float* sp = smem + output_body<MODE, NC>();         // [NH][64 j][PP]
    float* edge = sp + NH * CT * PP;                    // PER_CHANNEL: [4][SL] the decays of a block of 16 tokens
    __shared__ float s_a[NH][CT], s_cum[NH][CT], s_b[NH][CT];
    grid_dep_launch();
    grid_dep_wait();
    const int c = blockIdx.x, h = blockIdx.y * NH, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int dvv = ONES ? p.dv - 1 : p.dv, col0 = blockIdx.z * 64 * NC, nv = NH == 2 ? dvv : min(64 * NC, dvv - col0);
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.qk_group;
    if (c == 0)                                         // rows behind the last sequence belong to nobody: a defined value
        for (int t = p.chunk_start[p.n_chunks]; t < p.T_rows; ++t) {
            for (int e = tid; e < NH * nv; e += THREADS) p.o[(size_t)t * p.ldo + (size_t)(h + e / nv) * p.dv + (NH == 2 ? 0 : col0) + e % nv] = 0.f;
            if (ONES && col0 == 0 && tid == 0) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + dvv] = 0.f;
        }
    if (n <= 0) return;
    if (n > CT) {
        for (int x = 0; x < NH; ++x) {
            float* S = p.chunk_state + ((size_t)c * p.H + h + x) * p.dk * p.dvp;
            walk_in_order<TI, MODE>(p, S, c, h + x, col0, nv, true);
            if (ONES && col0 == 0) walk_in_order<TI, MODE>(p, S, c, h + x, dvv, 1, true);
        }
        return;
    }
    if (!PER_CHANNEL) {                                 // the tokens' decays and weights
        for (int e = tid; e < NH * CT; e += THREADS) {
            const int x = e / CT, t = e % CT;
            s_a[x][t] = t < n ? decay_at<MODE>(p, t0 + t, h + x, 0) : (MODE == 5 ? 0.f : 1.f);
            s_b[x][t] = t >= n ? 0.f : (MODE == 2 || MODE == 5) ? p.gb[(size_t)(t0 + t) * p.ldg + h + x] : 1.f;
        }
    }
    f32x2 acc[8][2 * NC], raw[8][2];
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        raw[i][0] = raw[i][1] = 0ull;
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;
    }
    float ones_part = 0.f;                              // ONES: q_t . S0's last column, token tid
    if (PER_CHANNEL)
        for (int e = tid; e < CT * PP; e += THREADS) sp[e] = 0.f;

    // q and k of a slice on their way to registers; the states' slice on its way to shared memory
    Raw4<TI> rq[NQ], rk[NQ];
    constexpr int LANES = SL / 4;                       // lanes that share a token's slice; a warp writes every bank of the staged tile once
    auto token_of = [&](int e) { return PER_CHANNEL ? e / LANES : (e >> 5) * 4 + ((e & 31) >> 3); };
    auto channel_of = [&](int e) { return PER_CHANNEL ? (e % LANES) * 4 : (e & 7) * 4; };
    auto fetch = [&](int i0) {
        const int nk = min(SL, p.dk - i0);
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS, t = token_of(e), i = channel_of(e);
            get_four(rq[x], (const TI*)p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, t < n, p.vec_q);
            get_four(rk[x], (const TI*)p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, t < n, p.vec_k);
        }
    };
    auto fetch_state = [&](int i0, float* dst) {
        const int nk = min(SL, p.dk - i0);
#pragma unroll 4
        for (int e = tid; e < SL * 16 * NC; e += THREADS) {
            const int i = e / (16 * NC), col = (e % (16 * NC)) * 4, x = NH == 2 ? col >> 6 : 0, own = NH == 2 ? col & 63 : col0 + col;
            copy16(dst + e * 4, p.chunk_state + (((size_t)c * p.H + h + x) * p.dk + i0 + i) * p.dvp + own, i < nk && own < dvv);
        }
    };
    fetch(0);
    if (!PER_CHANNEL) {
        fetch_state(0, ss);
        __syncthreads();
        for (int e = tid; e < NH * CT; e += THREADS) {  // the decays between two tokens, with the earlier one's weight; those since the start
            const int x = e / CT, j = e % CT;
            float w = s_b[x][j], cum = 1.f;
#pragma unroll 8
            for (int t = 0; t < CT; ++t) {
                const float a = s_a[x][t];
                if (t > j) w = times_decay<MODE>(w, a);
                if (t <= j) cum = times_decay<MODE>(cum, a);
                sp[(x * CT + j) * PP + t] = t >= j ? w : 0.f;
            }
            s_cum[x][j] = cum;
        }
    }
    for (int i0 = 0; i0 < p.dk; i0 += SL) {
        const int nk = min(SL, p.dk - i0);
        float* const s_now = PER_CHANNEL ? ss : ss + (i0 / SL & 1) * SL * COLS;
        __syncthreads();
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS, t = token_of(e), i = channel_of(e);
            const float4 q4 = rq[x].value(), k4 = rk[x].value();
            const float fq[4] = {q4.x, q4.y, q4.z, q4.w}, fk[4] = {k4.x, k4.y, k4.z, k4.w};
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                sq[at_ct(i + y, t)] = WKV ? fq[y] : fq[y] * p.q_scale;
                sk[at_ct(i + y, t)] = fk[y];
            }
            if (PER_CHANNEL) {
#pragma unroll
                for (int y = 0; y < 4; ++y) sw[at_ct(i + y, t)] = t < n && i + y < nk ? decay_at<MODE>(p, t0 + t, h, i0 + i + y) : 1.f;
            }
        }
        if (!PER_CHANNEL) {
            copies_done();
            __syncthreads();
            if (i0 + SL < p.dk) {
                fetch_state(i0 + SL, ss + ((i0 / SL + 1) & 1) * SL * COLS);
                fetch(i0 + SL);
            }
            // q k^T and q S0 of this slice
#pragma unroll 4
            for (int k = 0; k < SL; ++k) {
                const float4 x = *reinterpret_cast<const float4*>(sq + at_ct(k, ty * 4)), y = *reinterpret_cast<const float4*>(sq + at_ct(k, 32 + ty * 4));
                const float a[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
                const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(sk + at_ct(k, tx * 4));
                f32x2 b[2 * NC];
#pragma unroll
                for (int g = 0; g < NC; ++g) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(s_now + k * COLS + g * 64 + tx * 4);
                    b[2 * g] = w.x;
                    b[2 * g + 1] = w.y;
                }
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                    const f32x2 aa = pack2(a[i], a[i]);
                    raw[i][0] = fma2(aa, kk.x, raw[i][0]);
                    raw[i][1] = fma2(aa, kk.y, raw[i][1]);
#pragma unroll
                    for (int j = 0; j < 2 * NC; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
                }
            }
            if (ONES && blockIdx.z == 0 && tid < CT) {
                const float* last = p.chunk_state + (((size_t)c * p.H + h) * p.dk + i0) * p.dvp + dvv;
                for (int i = 0; i < nk; ++i) ones_part = fmaf(sq[at_ct(i, tid)], last[(size_t)i * p.dvp], ones_part);
            }
        } else {
            __syncthreads();
            // pairs of tokens within a block of 16, a warp per block: lane = token j and half of the channels
            const int blk = tid >> 5, lane = tid & 31, jj = lane & 15, b0 = blk * 16;
            {
                float d[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) d[x] = 0.f;
                for (int i = (lane >> 4) * (SL / 2); i < (lane >> 4) * (SL / 2) + SL / 2; ++i) {
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
                for (int x = 0; x < 16; ++x) {
                    const float sum = d[x] + __shfl_xor_sync(0xffffffffu, d[x], 16);
                    if (lane < 16 && x >= jj) sp[(b0 + jj) * PP + b0 + x] += sum;
                }
            }
            __syncthreads();
            // q times the decays since the start of its block of 16, k times those up to the block's end, the block's whole decay
            for (int e = tid; e < SL * 4; e += THREADS) {        // neighbouring lanes four channels apart: other banks
                const int i = (e & 15) * 4 + (e >> 4 & 3), g = e >> 6;
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
            // a block's tokens against all earlier ones, whose k are taken on to this block's start; a warp has 16 of the channels
            f32x2 x1[2][2], x2[4][2], x3[6][2];
#pragma unroll
            for (int x = 0; x < 6; ++x) {
                if (x < 2) x1[x][0] = x1[x][1] = 0ull;
                if (x < 4) x2[x][0] = x2[x][1] = 0ull;
                x3[x][0] = x3[x][1] = 0ull;
            }
            const int ch = blk * 16 + (jj & 3) * 4 + (jj >> 2), eighth = (lane >> 4) * 8;
            cross_product<1, 16, at_ct>(x1, sq, sk, blk * 16, lane);
            __syncwarp();
#pragma unroll
            for (int x = 0; x < 2; ++x) scale_four(sk + at_ct(ch, eighth + 4 * x), edge[SL + ch]);
            __syncwarp();
            cross_product<2, 16, at_ct>(x2, sq, sk, blk * 16, lane);
            __syncwarp();
#pragma unroll
            for (int x = 0; x < 4; ++x) scale_four(sk + at_ct(ch, 2 * eighth + 4 * x), edge[2 * SL + ch]);
            __syncwarp();
            cross_product<3, 16, at_ct>(x3, sq, sk, blk * 16, lane);
            __syncthreads();
            // the warps' sums over k and the decays, then added up; q times the decays since the chunk's start
            cross_store<1>(sk + blk * CROSS, x1, lane);
            cross_store<2>(sk + blk * CROSS, x2, lane);
            cross_store<3>(sk + blk * CROSS, x3, lane);
            for (int e = tid; e < SL * 12; e += THREADS) {
                const int i = (e & 15) * 4 + (e >> 4 & 3), t = 16 + (e >> 6) * 4;
                float x = 1.f;
                for (int m = 0; m < t / 16; ++m) x *= edge[m * SL + i];
                scale_four(sq + at_ct(i, t), x);
            }
            __syncthreads();
#pragma unroll
            for (int pair = 0; pair < 6; ++pair) {      // blocks (1,0) (2,0) (2,1) (3,0) (3,1) (3,2)
                const int I = pair == 0 ? 1 : pair < 3 ? 2 : 3, J = pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3;
                for (int e = tid; e < 256; e += THREADS) {
                    const int t = e & 15, j = J * 16 + (e >> 4);
                    const float* at = sk + cross_at(I) + t * (16 * I + 1) + j;
                    sp[j * PP + I * 16 + t] += (at[0] + at[CROSS]) + (at[2 * CROSS] + at[3 * CROSS]);
                }
            }
            __syncthreads();
            fetch_state(i0, ss);                        // over k and the decays
            if (i0 + SL < p.dk) fetch(i0 + SL);
            copies_done();
            __syncthreads();
            tile_product<NC, true>(acc, sq, ss, SL, ty, tx);
        }
    }
    Raw4<TI> rv[NV];
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const int e = tid + x * THREADS, j = e / (16 * NC), col = (e % (16 * NC)) * 4, head = NH == 2 ? col >> 6 : 0, own = NH == 2 ? col & 63 : col;
        get_four(rv[x], (const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)(h + head) * dvv + (NH == 2 ? 0 : col0), own, nv, j < n, p.vec_v);
    }
    __syncthreads();
    // the weights P[j][t], and acc times the decays since the chunk's start
    if (!PER_CHANNEL) {
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const int t = (i >> 2) * 32 + ty * 4 + (i & 3);
            const float2 r0 = unpack2(raw[i][0]), r1 = unpack2(raw[i][1]);
#pragma unroll
            for (int x = 0; x < NH; ++x) {
                float* w = sp + (x * CT + tx * 4) * PP + t;
                // a weight of zero stays zero whatever the product is: a token's q never meets a later token's k
                w[0] = tx * 4 <= t ? w[0] * r0.x : 0.f; w[PP] = tx * 4 + 1 <= t ? w[PP] * r0.y : 0.f;
                w[2 * PP] = tx * 4 + 2 <= t ? w[2 * PP] * r1.x : 0.f; w[3 * PP] = tx * 4 + 3 <= t ? w[3 * PP] * r1.y : 0.f;
            }
#pragma unroll
            for (int j = 0; j < 2 * NC; ++j) {
                const float cum = s_cum[NH == 2 ? j >> 1 : 0][t];
                acc[i][j] = mul2(pack2(cum, cum), acc[i][j]);
            }
        }
    }
    bool odd = false;                                   // a value that is not finite must not meet the weights of zero of earlier tokens
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const float4 f = rv[x].value();
        odd |= !(fabsf(f.x) <= 3.402823466e38f && fabsf(f.y) <= 3.402823466e38f && fabsf(f.z) <= 3.402823466e38f && fabsf(f.w) <= 3.402823466e38f);
        *reinterpret_cast<float4*>(svv + (tid + x * THREADS) * 4) = f;
    }
    odd = __syncthreads_or(odd);
    if (odd) add_values<NC, NH, true>(acc, sp, svv, n, ty, tx);
    else add_values<NC, NH, false>(acc, sp, svv, n, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = (i >> 2) * 32 + ty * 4 + (i & 3);
        if (t >= n) continue;
#pragma unroll
        for (int g = 0; g < NC; ++g) {
            const int own = NH == 2 ? tx * 4 : g * 64 + tx * 4;
            float* dst = p.o + (size_t)(t0 + t) * p.ldo + (size_t)(NH == 2 ? h + g : h) * p.dv + (NH == 2 ? 0 : col0) + own;
            const float2 a = unpack2(acc[i][2 * g]), b = unpack2(acc[i][2 * g + 1]);
            if (p.vec_o && own < nv) *reinterpret_cast<float4*>(dst) = make_float4(a.x, a.y, b.x, b.y);
            else {
                if (own < nv) dst[0] = a.x;
                if (own + 1 < nv) dst[1] = a.y;
                if (own + 2 < nv) dst[2] = b.x;
                if (own + 3 < nv) dst[3] = b.y;
            }
        }
    }
    if (ONES && blockIdx.z == 0 && tid < n) {
        float sum = s_cum[0][tid] * ones_part;
        for (int j = 0; j <= tid; ++j) sum += sp[j * PP + tid];
        p.o[(size_t)(t0 + tid) * p.ldo + (size_t)h * p.dv + dvv] = sum;
    }
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

// One output by multiply-adds, where the tensor unit gave no number.  The weights are taken from their terms at `tp` where they have some.
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
        if (!is_number(w)) {
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
        if (!is_number(sum)) sum = plain_output<TI, MODE>(p, S, s_a[0], s_b[0], s_cum[0][tid], tp, h, t0, tid, dvv);
        p.o[(size_t)(t0 + tid) * p.ldo + (size_t)h * p.dv + dvv] = sum;
    }
    if (ok) ok = wait_done(&done, slices & 1, p.status);
    tc_fence_after_sync();
    take_sums<32>(out, own + head * 64, false);
    float* const o = p.o + (size_t)t0 * p.ldo + (size_t)(h + head) * p.dv + col;
    if (col < dvv) {
        const int rows = n - half * 32;
        bool odd = false;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            odd |= !is_number(out[x]);
            if (x < rows) o[(size_t)(half * 32 + x) * p.ldo] = out[x];
        }
        if (odd)
            for (int t = half * 32; t < min(n, half * 32 + 32); ++t)
                if (!is_number(o[(size_t)t * p.ldo])) o[(size_t)t * p.ldo] = plain_output<TI, MODE>(p, S, s_a[head], s_b[head], s_cum[head][t], tp + head * 3 * TILE, h + head, t0, t, col);
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

// NC: columns in 64s of a block (per channel), NH: heads of a block (one decay per head)
template <typename TI, int MODE, int NC, int NH>
int launch_output(const Scan& p, int n_chunks, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    cudaError_t e;
    if constexpr (MODE == 1 || MODE == 4) {
        const size_t smem = (size_t)(output_body<MODE, NC>() + NH * CT * (CT + 4) + 4 * 64) * sizeof(float);
        e = cudaFuncSetAttribute(chunk_output_kernel<TI, MODE, NC, NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e == cudaSuccess)
            e = qs_launch_dependent(chunk_output_kernel<TI, MODE, NC, NH>, dim3(n_chunks, p.H / NH, (dvv + 64 * NC - 1) / (64 * NC)), dim3(THREADS), smem, stream, p);
    } else {
        constexpr int smem = tile_smem<TI, NH>();
        const auto kernel = p.dk > 128 ? tile_output_kernel<TI, MODE, NH, true> : tile_output_kernel<TI, MODE, NH, false>;
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (e == cudaSuccess)
            e = qs_launch_dependent(kernel, dim3(n_chunks, p.H / NH, NH == 2 ? 1 : (dvv + 127) / 128), dim3(TILE_THREADS), smem, stream, p);
    }
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "state_scan, chunk outputs: %s", cudaGetErrorString(e));
    return qs_check_launch("state_scan, chunk outputs");
}

template <typename TI, int MODE>
int run(const Scan& p, int n_chunks, bool outputs, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    if (!outputs) return launch_added<TI, MODE>(p, n_chunks, stream);
    if constexpr (MODE == 5)                            // two heads that share q and k: their products once
        if (dvv <= 64 && p.qk_group % 2 == 0) return launch_output<TI, MODE, 2, 2>(p, n_chunks, stream);
    return dvv > 64 ? launch_output<TI, MODE, 2, 1>(p, n_chunks, stream) : launch_output<TI, MODE, MODE == 1 || MODE == 4 ? 1 : 2, 1>(p, n_chunks, stream);
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
                   long long ldg, float q_scale, int qk_group, float decay_scale, int32_t* status, cudaStream_t stream) {
    const size_t item = dtype == QS_F32 ? 4 : 2;
    auto fours = [&](const void* ptr, long long ld, int per_head) { return (int)(per_head % 4 == 0 && ld % 4 == 0 && ((uintptr_t)ptr % (4 * item)) == 0); };
    Scan p = {};
    p.q = q; p.k = k; p.v = v; p.ldq = (size_t)ldq; p.ldk = (size_t)ldk; p.ldv = (size_t)ldv;
    p.dlog = dlog; p.ldd = (size_t)ldd; p.head_decay = head_decay; p.ga = ga; p.gb = gb; p.ldg = (size_t)ldg;
    p.bonus = bonus; p.bonus_dtype = bonus_dtype; p.chunk_start = chunk_start; p.chunk_state = chunk_state; p.chunk_decay = chunk_decay;
    p.o = o; p.ldo = (size_t)ldo; p.H = H; p.dk = dk; p.dv = dv; p.dvp = (dv + 3) / 4 * 4; p.qk_group = qk_group;
    p.q_scale = q_scale; p.decay_scale = decay_scale;
    p.vec_q = fours(q, ldq, dk); p.vec_k = fours(k, ldk, dk); p.vec_v = fours(v, ldv, mode == 2 ? dv - 1 : dv);
    p.vec_o = mode != 2 && dv % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)o % 16) == 0;
    p.n_chunks = n_chunks; p.T_rows = T_rows; p.status = status;
    return dtype == QS_F32 ? pick<float>(mode, p, n_chunks, outputs != 0, stream) : pick<__nv_bfloat16>(mode, p, n_chunks, outputs != 0, stream);
}
