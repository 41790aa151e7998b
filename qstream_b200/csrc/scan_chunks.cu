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
// All arithmetic is 32-bit on the CUDA cores (paired multiply-adds).  Decays enter as products of at most 64 factors up to
// one, never as quotients, so small ones cost no precision: per token and head by a recursion down the columns of P; per
// channel in blocks of 16 tokens, a block's own pairs walked in order, pairs of blocks through the products up to the
// blocks' common edge.
//
// Bound by multiply-add issue with 16-byte shared-memory reads beside it.  The walk with a state column pair per thread that
// stood here before spent three operands from shared memory and a shuffle round per token and column pair:
// MEASURED_LINES
#include "scan.cuh"

namespace {

constexpr int CT = 64;                                  // tokens of a chunk
constexpr int THREADS = 128;

// Where channel c's column of a staged [channels][64 tokens] tile lies: tokens in groups of four, permuted by the channel's
// group of four, so that a warp that writes 8 x 4 channels of four tokens meets every bank once.
__device__ __forceinline__ int at_ct(int c, int t) { return c * CT + (t ^ (((c >> 2) & 7) << 2)); }
// The same for [channels][columns] tiles written by four lanes per column (16 channels) and eight columns per warp.
__device__ __forceinline__ int at_kc(int k, int col, int cols) { return k * cols + (col ^ (((k >> 2) & 3) << 3)); }

struct Scan {
    const void *q, *k, *v;
    size_t ldq, ldk, ldv;
    const float *dlog; size_t ldd;                      // per channel: logits of the decays
    const float *head_decay;                            // one decay per head
    const float *ga, *gb; size_t ldg;                   // per token and head: decays (less one in mode 5), input weights
    const void* bonus; int bonus_dtype;
    const int32_t* chunk_start;
    float *chunk_state, *chunk_decay;                   // [chunks][H][dv][dk], [chunks][H][dk]
    float* o; size_t ldo;
    int H, dk, dv, in_act, qk_group, n_chunks, T_rows;
    float q_scale, decay_scale;
    int vec_q, vec_k, vec_v, vec_s, vec_o;              // whether rows may be read (written) in pieces of four
};

// The decay of channel i of head h at row t, as a factor (mode 5: less one).
template <int MODE>
__device__ __forceinline__ float decay_at(const Scan& p, size_t t, int h, int i) {
    if (MODE == 0) return p.head_decay[h];
    if (MODE == 2 || MODE == 5) return p.ga[t * p.ldg + h];
    const float z = p.dlog[t * p.ldd + (size_t)h * p.dk + i];
    return MODE == 1 ? expf(-expf(z)) : expf(log_sigmoid_f32(z) * p.decay_scale);
}
template <int MODE>
__device__ __forceinline__ float times_decay(float x, float a) { return MODE == 5 ? fmaf(x, a, x) : x * a; }

// Four channels of a row from channel i on, zeros behind the last.
template <typename TI>
__device__ __forceinline__ void load_four(const TI* __restrict__ row, int i, int n, int vec, float (&f)[4]) {
    f[0] = f[1] = f[2] = f[3] = 0.f;
    if (i >= n) return;
    if (vec) {
        if constexpr (sizeof(TI) == 4) {
            const float4 x = *reinterpret_cast<const float4*>(row + i);
            f[0] = x.x; f[1] = x.y; f[2] = x.z; f[3] = x.w;
        } else {
            const uint2 u = *reinterpret_cast<const uint2*>(row + i);
            f[0] = __uint_as_float(u.x << 16); f[1] = __uint_as_float(u.x & 0xffff0000u);
            f[2] = __uint_as_float(u.y << 16); f[3] = __uint_as_float(u.y & 0xffff0000u);
        }
        return;
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) if (i + j < n) f[j] = to_f32(row[i + j]);
}

// A chunk of more than 64 tokens (the callers cut none): this block's columns of the state walked in order in global memory.
template <typename TI, int MODE>
__device__ void walk_in_order(const Scan& p, float* __restrict__ S, int c, int h, int col0, int cols, bool output) {
    constexpr bool ONES = MODE == 2, WKV = MODE == 1;
    const int t0 = p.chunk_start[c], t1 = p.chunk_start[c + 1], hq = h / p.qk_group, dvv = ONES ? p.dv - 1 : p.dv;
    for (int col = col0 + (int)threadIdx.x; col < col0 + cols; col += THREADS) {
        float* s = S + (size_t)col * p.dk;
        for (int t = t0; t < t1; ++t) {
            const TI* qr = (const TI*)p.q + (size_t)t * p.ldq + hq * p.dk;
            const TI* kr = (const TI*)p.k + (size_t)t * p.ldk + hq * p.dk;
            const float v = ONES && col == dvv ? 1.f : apply_activation(to_f32(((const TI*)p.v)[(size_t)t * p.ldv + (size_t)h * dvv + col]), p.in_act);
            const float b = MODE == 2 || MODE == 5 ? p.gb[(size_t)t * p.ldg + h] : 1.f;
            float o = 0.f;
            for (int i = 0; i < p.dk; ++i) {
                const float q = apply_activation(to_f32(qr[i]), p.in_act) * (WKV ? 1.f : p.q_scale);
                const float kv = apply_activation(to_f32(kr[i]), p.in_act) * b * v, a = decay_at<MODE>(p, t, h, i);
                const float before = s[i], after = times_decay<MODE>(before, a) + kv;
                o = fmaf(q, WKV ? fmaf(load_as_f32(p.bonus, p.bonus_dtype, (size_t)h * p.dk + i), kv, before) : after, o);
                s[i] = after;
            }
            if (output) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + col] = o;
        }
    }
}

// acc[8][4 NC] += A[k][8 rows] B[k][4 NC columns] over k < n: A a swizzled [k][64] tile (rows 4 ty .. and 32 + 4 ty ..), B rows of
// `cols` columns (4 tx .. of every 64).  `skew_b`: B is swizzled as by at_kc.
template <int NC, bool SKEW_B>
__device__ __forceinline__ void tile_product(f32x2 (&acc)[8][2 * NC], const float* __restrict__ A, const float* __restrict__ B, int n, int ty, int tx) {
#pragma unroll 4
    for (int k = 0; k < n; ++k) {
        const float4 x = *reinterpret_cast<const float4*>(A + at_ct(k, ty * 4)), y = *reinterpret_cast<const float4*>(A + at_ct(k, 32 + ty * 4));
        const float a[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
        f32x2 b[2 * NC];
#pragma unroll
        for (int g = 0; g < NC; ++g) {
            const int col = g * 64 + tx * 4;
            const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(B + (SKEW_B ? at_kc(k, col, 64 * NC) : k * 64 * NC + col));
            b[2 * g] = w.x;
            b[2 * g + 1] = w.y;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
            for (int j = 0; j < 2 * NC; ++j) acc[i][j] = fma2(aa, b[j], acc[i][j]);
        }
    }
}

// ----------------------------------------------------------------------------- what a chunk adds

// A block takes 64 value columns x up to 128 key channels of one head's state: added[col][i] = sum_j v_j[col] kw_j[i], tokens on
// the sum's side.  kw_j = k_j times the decays behind token j (per channel), or v_j carries them (per head).
template <typename TI, int MODE, int NC>
__global__ void __launch_bounds__(THREADS)
added_state_kernel(Scan p) {
    constexpr bool PER_CHANNEL = MODE == 1 || MODE == 4, ONES = MODE == 2;
    extern __shared__ __align__(16) float smem[];
    float* sv = smem;                                   // [tokens][64], swizzled as at_ct(token, column)
    float* sk = sv + CT * CT;                           // [tokens][64 NC]
    float* part = sk + CT * 64 * NC;                    // PER_CHANNEL: [parts][64 NC]
    __shared__ float s_a[CT], s_w[CT];
    grid_dep_launch();
    grid_dep_wait();
    const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int dk_tiles = (p.dk + 64 * NC - 1) / (64 * NC), col0 = blockIdx.z / dk_tiles * CT, i0 = blockIdx.z % dk_tiles * 64 * NC;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.qk_group;
    const int dvv = ONES ? p.dv - 1 : p.dv, nk = min(64 * NC, p.dk - i0), nv = min(CT, dvv - col0);
    float* added = p.chunk_state + ((size_t)c * p.H + h) * p.dv * p.dk;
    float* decays = p.chunk_decay + ((size_t)c * p.H + h) * p.dk;
    if (n > CT) {
        if (i0 == 0) {
            const int cols = col0 == 0 && ONES ? nv + 1 : nv;
            for (int e = tid; e < cols * p.dk; e += THREADS) added[((size_t)(e / p.dk < nv ? col0 + e / p.dk : dvv)) * p.dk + e % p.dk] = 0.f;
            __syncthreads();
            walk_in_order<TI, MODE>(p, added, c, h, col0, nv, false);
            if (ONES && col0 == 0) walk_in_order<TI, MODE>(p, added, c, h, dvv, 1, false);
            if (col0 == 0)
                for (int i = tid; i < p.dk; i += THREADS) {
                    float a = 1.f;
                    for (int t = t0; t < t0 + n; ++t) a = times_decay<MODE>(a, decay_at<MODE>(p, t, h, i));
                    decays[i] = a;
                }
        }
        return;
    }
    if (!PER_CHANNEL) {
        if (tid < CT) s_a[tid] = tid < n ? decay_at<MODE>(p, t0 + tid, h, 0) : (MODE == 5 ? 0.f : 1.f);
        __syncthreads();
        if (tid < CT) {                                 // the decays behind token tid, and its weight
            float w = 1.f;
            for (int t = CT - 1; t > tid; --t) w = times_decay<MODE>(w, s_a[t]);
            const float whole = times_decay<MODE>(w, s_a[tid]);
            if (MODE == 2 || MODE == 5) w *= tid < n ? p.gb[(size_t)(t0 + tid) * p.ldg + h] : 0.f;
            s_w[tid] = w;
            if (tid == 0) part[0] = whole;
        }
        __syncthreads();
        if (col0 == 0)
            for (int i = tid; i < nk; i += THREADS) decays[i0 + i] = part[0];
    }
    // values: token rows in pieces of four columns
    for (int e = tid; e < CT * 16; e += THREADS) {
        const int j = e >> 4, col = (e & 15) * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (j < n) {
            load_four((const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)h * dvv + col0, col, nv, p.vec_v, f);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (p.in_act) f[x] = apply_activation(f[x], p.in_act);
                if (!PER_CHANNEL) f[x] *= s_w[j];
                if (col + x >= nv) f[x] = 0.f;
            }
        }
        *reinterpret_cast<float4*>(sv + at_ct(j, col)) = make_float4(f[0], f[1], f[2], f[3]);
    }
    for (int e = tid; e < CT * 16 * NC; e += THREADS) {
        const int j = e / (16 * NC), i = (e - j * 16 * NC) * 4;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (j < n) {
            load_four((const TI*)p.k + (size_t)(t0 + j) * p.ldk + hq * p.dk + i0, i, nk, p.vec_k, f);
            if (p.in_act) {
#pragma unroll
                for (int x = 0; x < 4; ++x) f[x] = i + x < nk ? apply_activation(f[x], p.in_act) : 0.f;
            }
        }
        *reinterpret_cast<float4*>(sk + j * 64 * NC + i) = make_float4(f[0], f[1], f[2], f[3]);
    }
    if (PER_CHANNEL) {                                  // a thread takes a channel and a part of the tokens, from the last back
        constexpr int PARTS = NC == 1 ? 2 : 1, LEN = CT / PARTS;
        __syncthreads();
        const int i = tid % (64 * NC), g = tid / (64 * NC);
        float run = 1.f;
        for (int base = LEN - 16; base >= 0; base -= 16) {
            float a[16];
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                const int t = g * LEN + base + x;
                a[x] = t < n && i < nk ? decay_at<MODE>(p, t0 + t, h, i0 + i) : 1.f;
            }
#pragma unroll
            for (int x = 15; x >= 0; --x) {
                sk[(g * LEN + base + x) * 64 * NC + i] *= run;
                run *= a[x];
            }
        }
        part[g * 64 * NC + i] = run;
        __syncthreads();
        if (PARTS == 2 && g == 0) {
            const float later = part[64 * NC + i];
#pragma unroll 8
            for (int t = 0; t < LEN; ++t) sk[t * 64 * NC + i] *= later;
            run *= later;
        }
        if (g == 0 && i < nk && col0 == 0) decays[i0 + i] = run;
    }
    __syncthreads();
    f32x2 acc[8][2 * NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;
    tile_product<NC, false>(acc, sv, sk, n, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int col = (i >> 2) * 32 + ty * 4 + (i & 3);
        if (col >= nv) continue;
        float* row = added + (size_t)(col0 + col) * p.dk + i0;
#pragma unroll
        for (int g = 0; g < NC; ++g) {
            const int at = g * 64 + tx * 4;
            const float2 a = unpack2(acc[i][2 * g]), b = unpack2(acc[i][2 * g + 1]);
            if (p.vec_s && at < nk) *reinterpret_cast<float4*>(row + at) = make_float4(a.x, a.y, b.x, b.y);
            else {
                if (at < nk) row[at] = a.x;
                if (at + 1 < nk) row[at + 1] = a.y;
                if (at + 2 < nk) row[at + 2] = b.x;
                if (at + 3 < nk) row[at + 3] = b.y;
            }
        }
    }
    if (ONES && col0 == 0)                              // the column whose values are ones
        for (int i = tid; i < nk; i += THREADS) {
            float sum = 0.f;
            for (int j = 0; j < n; ++j) sum = fmaf(s_w[j], sk[j * 64 * NC + i], sum);
            added[(size_t)dvv * p.dk + i0 + i] = sum;
        }
}

// ----------------------------------------------------------------------------- a chunk's outputs

// A block takes the 64 tokens of a chunk and 64 NC value columns: of one head, or (NH = 2) 64 of each of two neighbouring heads
// that share q and k, whose products q k^T are then taken once.  The key channels pass in slices through shared memory.
template <typename TI, int MODE, int NC, int NH>
__global__ void __launch_bounds__(THREADS)
chunk_output_kernel(Scan p) {
    constexpr bool PER_CHANNEL = MODE == 1 || MODE == 4, ONES = MODE == 2, WKV = MODE == 1;
    constexpr int SL = PER_CHANNEL ? 64 : 32;           // channels of a slice
    constexpr int PP = CT + 4;                          // pitch of the weights P[j][t]
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                                   // [SL][64 tokens]
    float* sk = sq + SL * CT;                           // [SL][64 tokens]
    float* sw = sk + SL * CT;                           // PER_CHANNEL: the decays [SL][64 tokens]; then the state lies over sk, sw
    float* ss = PER_CHANNEL ? sk : sw;                  // [SL][64 NC]: a slice of the states the chunk starts from
    float* svv = smem;                                  // [64 tokens][64 NC]: the values, after the last slice
    constexpr int STAGE = PER_CHANNEL ? (3 * SL * CT > SL * CT + SL * 64 * NC ? 3 * SL * CT : SL * CT + SL * 64 * NC) : 2 * SL * CT + SL * 64 * NC;
    constexpr int VALUES = CT * 64 * NC;
    float* sp = smem + (STAGE > VALUES ? STAGE : VALUES);       // [NH][64 j][PP]
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
            float* S = p.chunk_state + ((size_t)c * p.H + h + x) * p.dv * p.dk;
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

    for (int i0 = 0; i0 < p.dk; i0 += SL) {
        const int nk = min(SL, p.dk - i0);
        __syncthreads();
        // q and k: eight (sixteen) lanes share a token's slice, a warp writes every bank once
        constexpr int LANES = SL / 4;
        for (int e = tid; e < CT * LANES; e += THREADS) {
            const int t = PER_CHANNEL ? e / LANES : (e >> 5) * 4 + ((e & 31) >> 3), i = PER_CHANNEL ? (e % LANES) * 4 : (e & 7) * 4;
            float fq[4] = {0.f, 0.f, 0.f, 0.f}, fk[4] = {0.f, 0.f, 0.f, 0.f};
            if (t < n) {
                load_four((const TI*)p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, p.vec_q, fq);
                load_four((const TI*)p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, p.vec_k, fk);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                if (p.in_act) { fq[x] = apply_activation(fq[x], p.in_act); fk[x] = apply_activation(fk[x], p.in_act); }
                if (!WKV) fq[x] *= p.q_scale;
                if (i + x >= nk) fq[x] = fk[x] = 0.f;
                sq[at_ct(i + x, t)] = fq[x];
                sk[at_ct(i + x, t)] = fk[x];
            }
            if (PER_CHANNEL) {
#pragma unroll
                for (int x = 0; x < 4; ++x) sw[at_ct(i + x, t)] = t < n && i + x < nk ? decay_at<MODE>(p, t0 + t, h, i0 + i + x) : 1.f;
            }
        }
        auto stage_state = [&]() {
            for (int e = tid; e < 64 * NC * LANES; e += THREADS) {          // four lanes take 16 channels of a column
                const int col = (e / 4) % (64 * NC), i = (e / (4 * 64 * NC)) * 16 + (e & 3) * 4;
                const int x = NH == 2 ? col >> 6 : 0, own = NH == 2 ? col & 63 : col0 + col;
                float f[4] = {0.f, 0.f, 0.f, 0.f};
                if (own < dvv)
                    load_four(p.chunk_state + (((size_t)c * p.H + h + x) * p.dv + own) * p.dk + i0, i, nk, p.vec_s, f);
#pragma unroll
                for (int y = 0; y < 4; ++y) ss[at_kc(i + y, col, 64 * NC)] = f[y];
            }
        };
        if (!PER_CHANNEL) {
            stage_state();
            __syncthreads();
            // q k^T and q S0 of this slice
#pragma unroll 4
            for (int k = 0; k < SL; ++k) {
                const float4 x = *reinterpret_cast<const float4*>(sq + at_ct(k, ty * 4)), y = *reinterpret_cast<const float4*>(sq + at_ct(k, 32 + ty * 4));
                const float a[8] = {x.x, x.y, x.z, x.w, y.x, y.y, y.z, y.w};
                const ulonglong2 kk = *reinterpret_cast<const ulonglong2*>(sk + at_ct(k, tx * 4));
                f32x2 b[2 * NC];
#pragma unroll
                for (int g = 0; g < NC; ++g) {
                    const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(ss + at_kc(k, g * 64 + tx * 4, 64 * NC));
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
                const float* last = p.chunk_state + (((size_t)c * p.H + h) * p.dv + dvv) * p.dk + i0;
                for (int i = 0; i < nk; ++i) ones_part = fmaf(sq[at_ct(i, tid)], last[i], ones_part);
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
                        if (x >= jj) d[x] = fmaf(fq[x], WKV && x == jj ? u * kj : run, d[x]);
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
            for (int e = tid; e < SL * 4; e += THREADS) {
                const int i = e % SL, g = e / SL;
                float run = 1.f;
#pragma unroll
                for (int t = 0; t < 16; ++t) {
                    float* x = sq + at_ct(i, g * 16 + t);
                    const float a = sw[at_ct(i, g * 16 + t)];
                    if (!WKV) run *= a;
                    *x *= run;
                    if (WKV) run *= a;
                }
                edge[g * SL + i] = run;
                run = 1.f;
#pragma unroll
                for (int t = 15; t >= 0; --t) {
                    sk[at_ct(i, g * 16 + t)] *= run;
                    run *= sw[at_ct(i, g * 16 + t)];
                }
            }
            __syncthreads();
            // pairs of blocks: (1,0) (2,0) (2,1) (3,0) (3,1) (3,2), 256 pairs of tokens each; a warp takes eight tokens t against the 16 j
            // of a pair of blocks at a time, a thread one t and four j
            for (int e = blk; e < 12; e += 4) {
                const int pair = e >> 1, I = pair == 0 ? 1 : pair < 3 ? 2 : 3, J = pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3;
                const int t = I * 16 + (e & 1) * 8 + (lane >> 2) , j = J * 16 + (lane & 3) * 4;
                float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f;
                for (int i = 0; i < SL; ++i) {
                    float x = sq[at_ct(i, t)];
                    for (int m = J + 1; m < I; ++m) x *= edge[m * SL + i];
                    const float4 kk = *reinterpret_cast<const float4*>(sk + at_ct(i, j));
                    s0 = fmaf(x, kk.x, s0); s1 = fmaf(x, kk.y, s1); s2 = fmaf(x, kk.z, s2); s3 = fmaf(x, kk.w, s3);
                }
                sp[j * PP + t] += s0; sp[(j + 1) * PP + t] += s1; sp[(j + 2) * PP + t] += s2; sp[(j + 3) * PP + t] += s3;
            }
            __syncthreads();
            // q times the decays since the chunk's start; the state over k and the decays
            for (int e = tid; e < SL * 48; e += THREADS) {
                const int i = e % SL, t = 16 + e / SL;
                float x = 1.f;
                for (int m = 0; m < t / 16; ++m) x *= edge[m * SL + i];
                sq[at_ct(i, t)] *= x;
            }
            stage_state();
            __syncthreads();
            tile_product<NC, true>(acc, sq, ss, SL, ty, tx);
        }
    }
    __syncthreads();
    // the weights P[j][t], and acc times the decays since the chunk's start
    if (!PER_CHANNEL) {
        for (int e = tid; e < NH * CT; e += THREADS) {
            const int x = e / CT, j = e % CT;
            float w = s_b[x][j];
            for (int t = 0; t < CT; ++t) {
                if (t > j) w = times_decay<MODE>(w, s_a[x][t]);
                sp[(x * CT + j) * PP + t] = t >= j ? w : 0.f;
            }
            float cum = 1.f;
            for (int t = 0; t <= j; ++t) cum = times_decay<MODE>(cum, s_a[x][t]);
            s_cum[x][j] = cum;
        }
        __syncthreads();
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
    for (int e = tid; e < CT * 16 * NC; e += THREADS) {
        const int j = e / (16 * NC), col = (e - j * 16 * NC) * 4;
        const int x = NH == 2 ? col >> 6 : 0, own = NH == 2 ? col & 63 : col;
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (j < n) {
            load_four((const TI*)p.v + (size_t)(t0 + j) * p.ldv + (size_t)(h + x) * dvv + (NH == 2 ? 0 : col0), own, nv, p.vec_v, f);
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                if (p.in_act) f[y] = own + y < nv ? apply_activation(f[y], p.in_act) : 0.f;
                odd |= !(fabsf(f[y]) <= 3.402823466e38f);
            }
        }
        *reinterpret_cast<float4*>(svv + j * 64 * NC + col) = make_float4(f[0], f[1], f[2], f[3]);
    }
    odd = __syncthreads_or(odd);
    // tokens j: the first 32 meet every t, the others only the last 32
    auto add_values = [&](bool later_only) {
#pragma unroll 2
        for (int j = 0; j < n; ++j) {
            f32x2 b[2 * NC];
#pragma unroll
            for (int g = 0; g < NC; ++g) {
                const ulonglong2 w = *reinterpret_cast<const ulonglong2*>(svv + j * 64 * NC + g * 64 + tx * 4);
                b[2 * g] = w.x;
                b[2 * g + 1] = w.y;
            }
#pragma unroll
            for (int g = 0; g < 2; ++g) {
                if (g == 0 && j >= 32) continue;
#pragma unroll
                for (int x = 0; x < NH; ++x) {
                    const float4 w = *reinterpret_cast<const float4*>(sp + (x * CT + j) * PP + g * 32 + ty * 4);
                    const float a[4] = {w.x, w.y, w.z, w.w};
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        if (later_only && g * 32 + ty * 4 + i < j) continue;
                        const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
                        for (int y = 0; y < 2 * NC; ++y)
                            if (NH == 1 || (y >> 1) == x) acc[g * 4 + i][y] = fma2(aa, b[y], acc[g * 4 + i][y]);
                    }
                }
            }
        }
    };
    if (odd) add_values(true);
    else add_values(false);
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

template <typename TI, int MODE, int NC>
int launch_added(const Scan& p, int n_chunks, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    const size_t smem = (size_t)(CT * CT + CT * 64 * NC + 2 * 64 * NC) * sizeof(float);
    cudaError_t e = smem > 48 * 1024 ? cudaFuncSetAttribute(added_state_kernel<TI, MODE, NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) : cudaSuccess;
    const int tiles = ((dvv + CT - 1) / CT) * ((p.dk + 64 * NC - 1) / (64 * NC));
    if (e == cudaSuccess) e = qs_launch_dependent(added_state_kernel<TI, MODE, NC>, dim3(n_chunks, p.H, tiles), dim3(THREADS), smem, stream, p);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "state_scan, added states: %s", cudaGetErrorString(e));
    return qs_check_launch("state_scan, added states");
}

template <typename TI, int MODE, int NC, int NH>
int launch_output(const Scan& p, int n_chunks, cudaStream_t stream) {
    constexpr bool PER_CHANNEL = MODE == 1 || MODE == 4;
    constexpr int SL = PER_CHANNEL ? 64 : 32;
    constexpr int STAGE = PER_CHANNEL ? (3 * SL * CT > SL * CT + SL * 64 * NC ? 3 * SL * CT : SL * CT + SL * 64 * NC) : 2 * SL * CT + SL * 64 * NC;
    constexpr int VALUES = CT * 64 * NC;
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    const size_t smem = (size_t)((STAGE > VALUES ? STAGE : VALUES) + NH * CT * (CT + 4) + (PER_CHANNEL ? 4 * SL : 0)) * sizeof(float);
    cudaError_t e = cudaFuncSetAttribute(chunk_output_kernel<TI, MODE, NC, NH>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    const int tiles = NH == 2 ? 1 : (dvv + 64 * NC - 1) / (64 * NC);
    if (e == cudaSuccess)
        e = qs_launch_dependent(chunk_output_kernel<TI, MODE, NC, NH>, dim3(n_chunks, p.H / NH, tiles), dim3(THREADS), smem, stream, p);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "state_scan, chunk outputs: %s", cudaGetErrorString(e));
    return qs_check_launch("state_scan, chunk outputs");
}

template <typename TI, int MODE>
int run(const Scan& p, int n_chunks, bool outputs, cudaStream_t stream) {
    const int dvv = MODE == 2 ? p.dv - 1 : p.dv;
    if (!outputs) return p.dk > 64 ? launch_added<TI, MODE, 2>(p, n_chunks, stream) : launch_added<TI, MODE, 1>(p, n_chunks, stream);
    if constexpr (MODE == 5)                            // two heads that share q and k: their products once
        if (dvv <= 64 && dvv > 32 && p.qk_group % 2 == 0) return launch_output<TI, MODE, 2, 2>(p, n_chunks, stream);
    return dvv > 64 ? launch_output<TI, MODE, 2, 1>(p, n_chunks, stream) : launch_output<TI, MODE, 1, 1>(p, n_chunks, stream);
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

}  // namespace

// The first (outputs == 0: chunk_state becomes what every chunk adds, chunk_decay its decays) and the last kernel (chunk_state
// holds the states the chunks start from) of a scan in chunks; operands as for `qs_state_scan`.
int qs_scan_chunks(int mode, int outputs, float* o, long long ldo, const void* q, long long ldq, const void* k, long long ldk, const void* v, long long ldv,
                   int dtype, const float* dlog, long long ldd, const float* head_decay, const void* bonus, int bonus_dtype, int H, int dk, int dv,
                   int in_act, const int32_t* chunk_start, int n_chunks, int T_rows, float* chunk_state, float* chunk_decay, const float* ga, const float* gb,
                   long long ldg, float q_scale, int qk_group, float decay_scale, cudaStream_t stream) {
    const size_t item = dtype == QS_F32 ? 4 : 2;
    auto fours = [&](const void* ptr, long long ld, int per_head) { return (int)(per_head % 4 == 0 && ld % 4 == 0 && ((uintptr_t)ptr % (4 * item)) == 0); };
    Scan p = {};
    p.q = q; p.k = k; p.v = v; p.ldq = (size_t)ldq; p.ldk = (size_t)ldk; p.ldv = (size_t)ldv;
    p.dlog = dlog; p.ldd = (size_t)ldd; p.head_decay = head_decay; p.ga = ga; p.gb = gb; p.ldg = (size_t)ldg;
    p.bonus = bonus; p.bonus_dtype = bonus_dtype; p.chunk_start = chunk_start; p.chunk_state = chunk_state; p.chunk_decay = chunk_decay;
    p.o = o; p.ldo = (size_t)ldo; p.H = H; p.dk = dk; p.dv = dv; p.in_act = in_act; p.qk_group = qk_group;
    p.q_scale = q_scale; p.decay_scale = decay_scale;
    p.vec_q = fours(q, ldq, dk); p.vec_k = fours(k, ldk, dk); p.vec_v = fours(v, ldv, mode == 2 ? dv - 1 : dv);
    p.vec_o = mode != 2 && dv % 4 == 0 && ldo % 4 == 0 && ((uintptr_t)o % 16) == 0;
    p.n_chunks = n_chunks; p.T_rows = T_rows;
    p.vec_s = dk % 4 == 0 && ((uintptr_t)chunk_state % 16) == 0;
    return dtype == QS_F32 ? pick<float>(mode, p, n_chunks, outputs != 0, stream) : pick<__nv_bfloat16>(mode, p, n_chunks, outputs != 0, stream);
}
