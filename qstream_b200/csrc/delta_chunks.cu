// The gated delta rule over long prompts, chunks of up to 64 tokens as matrix products.
//
//   S' = diag(g_t) S,  u_t = beta_t (v_t - S'^T k_t),  S = S' + k_t u_t^T,  o_t = S^T q_t
//
// With G_t = g_1 .. g_t within a chunk that starts from S0, and for j <= t
//   A[t][j] = sum_i k_t[i] k_j[i] (g_{j+1} .. g_t)[i],   B[t][j] the same with q_t,
// the writes obey u_t = beta_t (v_t - (G_t k_t)^T S0 - sum_{j < t} A[t][j] u_j), a triangular system.  Solved once for the right
// sides beta v (U) and beta G k (W), it gives u = U - W S0, and
//   S_end = diag(G_n) S0 + sum_j (g_{j+1} .. g_n k_j) u_j^T,      o_t = (G_t q_t)^T S0 + sum_{j <= t} B[t][j] u_j.
//
//   delta_terms_kernel    per chunk and head, side by side: A and B (as for a decay per channel in scan_chunks.cu), the solution by
//                         substitution with a column pair per thread in registers, the decayed q and k
//   delta_walk_kernel     per sequence, head and 16 value columns, the chunks in order: u and the next state, two small products each
//   delta_output_kernel   per chunk and head, side by side: the outputs
//
// All 32-bit; decays only as products of factors up to one.  Three walks of every chunk token by token (what it does to an
// identity, what it writes from nothing, its outputs) and a product of dk x dk matrices in the prefix stood here before: 2,000 tokens, 16
// heads of 128 x 128, with their projections, convolutions and norms 1,678 us, now 532 (the terms 214, the walk 134, the outputs 59).
#include "scan.cuh"
#include "scan_tiles.cuh"

namespace {

constexpr int WC = 16;                                  // value columns of a block of the walk
constexpr int WALK = 256;

struct Delta {
    const float *q, *k, *v, *g, *beta;                  // rows of ldq, ldk, ldv, ldg, ldb
    size_t ldq, ldk, ldv, ldg, ldb;
    const int32_t *chunk_start, *seq_chunk, *seq_slot;
    float *W, *K, *Q;                                   // [chunks][H][64][dkp]: the solution's W, k times the decays behind it, q times those before
    float *U;                                           // [chunks][H][64][dvp]
    float *B;                                           // [chunks][H][64 j][64 t]
    float *decay;                                       // [chunks][H][dkp]
    float *start;                                       // [chunks][H][dk][dvp]: the states the chunks start from
    float *state; size_t slot_stride;
    float *o; size_t ldo;
    int H, dk, dv, dkp, dvp, group, n_chunks, T_rows;
    int vec_q, vec_k, vec_g;
};

// X[t] <- beta_t R[t] - sum_{j < t} (beta_t A[t][j]) X[j] for two columns per thread, the 64 tokens' values in registers.  minus [64][PP]
// holds -beta A; rows of R from `rows` on count as zero.
__device__ __noinline__ void substitute(float* __restrict__ X, int ldx, const float* R, size_t ldr, int cols, int rows, const float* __restrict__ minus,
                                        const float* __restrict__ beta) {
    for (int c = 2 * threadIdx.x; c < cols; c += 2 * THREADS) {
        f32x2 x[CT];
        const bool two = c + 1 < cols;
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const float a = t < rows ? R[(size_t)t * ldr + c] : 0.f, b = t < rows && two ? R[(size_t)t * ldr + c + 1] : 0.f;
            x[t] = pack2(a, b);
        }
#pragma unroll
        for (int t = 0; t < CT; ++t) {
            const float b = beta[t];
            f32x2 sum = mul2(pack2(b, b), x[t]);
#pragma unroll
            for (int j = 0; j < t; j += 4) {
                const float4 m = *reinterpret_cast<const float4*>(minus + t * PP + j);
                sum = fma2(pack2(m.x, m.x), x[j], sum);
                if (j + 1 < t) sum = fma2(pack2(m.y, m.y), x[j + 1], sum);
                if (j + 2 < t) sum = fma2(pack2(m.z, m.z), x[j + 2], sum);
                if (j + 3 < t) sum = fma2(pack2(m.w, m.w), x[j + 3], sum);
            }
            x[t] = sum;
            const float2 v = unpack2(sum);
            X[(size_t)t * ldx + c] = v.x;
            if (two) X[(size_t)t * ldx + c + 1] = v.y;
        }
    }
}

constexpr int SL = 64;                                  // key channels of a slice
constexpr int TERMS_SMEM = (3 * SL * CT + 2 * CT * PP + 4 * SL) * sizeof(float);

__global__ void __launch_bounds__(THREADS, 2)
delta_terms_kernel(Delta p) {
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                                   // [SL][64 tokens]
    float* sk = sq + SL * CT;
    float* sw = sk + SL * CT;                           // the decays; then k times the decays since its block's start
    float* sA = sw + SL * CT;                           // [64 t][PP]
    float* sB = sA + CT * PP;                           // [64 j][PP]
    float* edge = sB + CT * PP;                         // [4][SL] the decays of a block of 16 tokens
    __shared__ float s_beta[CT];
    grid_dep_launch();
    grid_dep_wait();
    const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.group;
    if (n <= 0 || n > CT) return;                       // longer chunks are walked token by token
    const size_t unit = (size_t)c * p.H + h;
    if (tid < CT) s_beta[tid] = tid < n ? p.beta[(size_t)(t0 + tid) * p.ldb + h] : 0.f;
    for (int e = tid; e < 2 * CT * PP; e += THREADS) sA[e] = 0.f;
    constexpr int FOURS = SL / 4, NQ = CT * FOURS / THREADS;
    for (int i0 = 0; i0 < p.dkp; i0 += SL) {
        const int nk = min(SL, p.dk - i0);
        Raw4<float> rq[NQ], rk[NQ], rg[NQ];
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS, t = e / FOURS, i = (e % FOURS) * 4;
            get_four(rq[x], p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, t < n, p.vec_q);
            get_four(rk[x], p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, t < n, p.vec_k);
            get_four(rg[x], p.g + (size_t)(t0 + t) * p.ldg + h * p.dk + i0, i, nk, t < n, p.vec_g);
        }
        __syncthreads();
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS, t = e / FOURS, i = (e % FOURS) * 4;
            const float4 a = rq[x].value(), b = rk[x].value(), d = rg[x].value();
            const float fq[4] = {a.x, a.y, a.z, a.w}, fk[4] = {b.x, b.y, b.z, b.w}, fg[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                sq[at_ct(i + y, t)] = fq[y];
                sk[at_ct(i + y, t)] = fk[y];
                sw[at_ct(i + y, t)] = t < n && i + y < nk ? fg[y] : 1.f;
            }
        }
        __syncthreads();
        // pairs of tokens within a block of 16, a warp per block: lane = token j and half of the channels
        {
            const int jj = lane & 15, b0 = warp * 16;
            float da[16], db[16];
#pragma unroll
            for (int x = 0; x < 16; ++x) da[x] = db[x] = 0.f;
            for (int i = (lane >> 4) * (SL / 2); i < (lane >> 4) * (SL / 2) + SL / 2; ++i) {
                float run = sk[at_ct(i, b0 + jj)];
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const float4 q4 = *reinterpret_cast<const float4*>(sq + at_ct(i, b0 + 4 * b)), k4 = *reinterpret_cast<const float4*>(sk + at_ct(i, b0 + 4 * b));
                    const float4 w4 = *reinterpret_cast<const float4*>(sw + at_ct(i, b0 + 4 * b));
                    const float fq[4] = {q4.x, q4.y, q4.z, q4.w}, fk[4] = {k4.x, k4.y, k4.z, k4.w}, fw[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                    for (int y = 0; y < 4; ++y) {
                        const int x = 4 * b + y;
                        if (x > jj) {
                            run *= fw[y];
                            da[x] = fmaf(fk[y], run, da[x]);
                        }
                        if (x >= jj) db[x] = fmaf(fq[y], run, db[x]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                const float a = da[x] + __shfl_xor_sync(0xffffffffu, da[x], 16), b = db[x] + __shfl_xor_sync(0xffffffffu, db[x], 16);
                if (lane < 16 && x >= jj) {
                    sB[(b0 + jj) * PP + b0 + x] += b;
                    if (x > jj) sA[(b0 + x) * PP + b0 + jj] += a;
                }
            }
        }
        __syncthreads();
        // q and k times the decays since the start of their block of 16, k times those up to the block's end, the block's whole decay
        for (int e = tid; e < SL * 4; e += THREADS) {
            const int i = e % SL, b = e / SL;
            float a[16], run = 1.f;
#pragma unroll
            for (int x = 0; x < 16; ++x) a[x] = sw[at_ct(i, b * 16 + x)];
#pragma unroll
            for (int x = 0; x < 16; ++x) {
                run *= a[x];
                sq[at_ct(i, b * 16 + x)] *= run;
                sw[at_ct(i, b * 16 + x)] = sk[at_ct(i, b * 16 + x)] * run;
            }
            edge[b * SL + i] = run;
            run = 1.f;
#pragma unroll
            for (int x = 15; x >= 0; --x) {
                sk[at_ct(i, b * 16 + x)] *= run;
                run *= a[x];
            }
        }
        __syncthreads();
        // pairs of blocks: (1,0) (2,0) (2,1) (3,0) (3,1) (3,2); a warp takes eight tokens t against the 16 j of a pair of blocks at a time
        for (int e = warp; e < 12; e += 4) {
            const int pair = e >> 1, I = pair == 0 ? 1 : pair < 3 ? 2 : 3, J = pair == 0 ? 0 : pair < 3 ? pair - 1 : pair - 3;
            const int t = I * 16 + (e & 1) * 8 + (lane >> 2), j = J * 16 + (lane & 3) * 4;
            float sa[4] = {0.f, 0.f, 0.f, 0.f}, sb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
            for (int i = 0; i < SL; ++i) {
                float d = 1.f;
                for (int m = J + 1; m < I; ++m) d *= edge[m * SL + i];
                const float x = sq[at_ct(i, t)] * d, y = sw[at_ct(i, t)] * d;
                const float4 kk = *reinterpret_cast<const float4*>(sk + at_ct(i, j));
                sb[0] = fmaf(x, kk.x, sb[0]); sb[1] = fmaf(x, kk.y, sb[1]); sb[2] = fmaf(x, kk.z, sb[2]); sb[3] = fmaf(x, kk.w, sb[3]);
                sa[0] = fmaf(y, kk.x, sa[0]); sa[1] = fmaf(y, kk.y, sa[1]); sa[2] = fmaf(y, kk.z, sa[2]); sa[3] = fmaf(y, kk.w, sa[3]);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                sB[(j + x) * PP + t] += sb[x];
                sA[t * PP + j + x] += sa[x];
            }
        }
        // the same relative to the chunk's ends, for the products with the states
        const int nw = min(SL, p.dkp - i0);
        for (int e = tid; e < CT * SL; e += THREADS) {
            const int i = e % SL, t = e / SL, b = t >> 4;
            if (i >= nw) continue;
            float before = 1.f, after = 1.f;
            for (int m = 0; m < b; ++m) before *= edge[m * SL + i];
            for (int m = b + 1; m < 4; ++m) after *= edge[m * SL + i];
            const size_t at = (unit * CT + t) * p.dkp + i0 + i;
            p.Q[at] = sq[at_ct(i, t)] * before;
            p.W[at] = sw[at_ct(i, t)] * before;
            p.K[at] = sk[at_ct(i, t)] * after;
            if (t == 0) p.decay[unit * p.dkp + i0 + i] = edge[i] * after;
        }
        __syncthreads();
    }
    for (int e = tid; e < CT * CT; e += THREADS) {
        const int r = e >> 6, j = e & 63;
        sA[r * PP + j] *= -s_beta[r];
        p.B[unit * CT * CT + e] = sB[r * PP + j];
    }
    __syncthreads();
    substitute(p.W + unit * CT * p.dkp, p.dkp, p.W + unit * CT * p.dkp, p.dkp, p.dk, CT, sA, s_beta);
    substitute(p.U + unit * CT * p.dvp, p.dvp, p.v + (size_t)t0 * p.ldv + (size_t)h * p.dv, p.ldv, p.dv, n, sA, s_beta);
}

__host__ __device__ inline int walk_stage(int dkp) { return CT * (dkp + 4) + CT * dkp; }       // W and K of a chunk
inline int walk_stages(int dkp) { return dkp <= 128 ? 2 : 1; }
inline size_t walk_smem(int dkp) {
    return (size_t)(walk_stages(dkp) * walk_stage(dkp) + dkp * WC + CT * WC + (4 * CT * WC > dkp * WC ? 4 * CT * WC : dkp * WC)) * sizeof(float);
}

__global__ void __launch_bounds__(WALK)
delta_walk_kernel(Delta p, int stages) {
    extern __shared__ __align__(16) float smem[];
    const int dkp = p.dkp, wp = dkp + 4;
    float* sS = smem + stages * walk_stage(dkp);        // [dk][16]
    float* sU = sS + dkp * WC;                          // [64][16]
    float* red = sU + CT * WC;                          // [4 parts][64][16], [dk][16]
    grid_dep_launch();
    grid_dep_wait();
    const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * WC, tid = threadIdx.x;
    const int slot = p.seq_slot[s], c0 = p.seq_chunk[s], c1 = p.seq_chunk[s + 1];
    if (slot < 0 || c1 <= c0) return;
    const int n_cols = min(WC, p.dv - col0);
    float* own = p.state + (size_t)slot * p.slot_stride + ((size_t)h * p.dv + col0) * p.dk;
    for (int e = tid; e < dkp * WC; e += WALK) {
        const int col = e / dkp, i = e - col * dkp;
        sS[i * WC + col] = col < n_cols && i < p.dk ? own[(size_t)col * p.dk + i] : 0.f;
    }
    auto fetch = [&](int c, int stage) {
        const int n = p.chunk_start[c + 1] - p.chunk_start[c];
        if (n <= 0 || n > CT) return;
        const size_t unit = (size_t)c * p.H + h;
        float* w = smem + stage * walk_stage(dkp);
        float* k = w + CT * wp;
        const int fours = dkp / 4;
        for (int e = tid; e < CT * fours; e += WALK) {
            const int t = e / fours, i = (e - t * fours) * 4;
            copy16(w + t * wp + i, p.W + (unit * CT + t) * dkp + i, true);
            copy16(k + t * dkp + i, p.K + (unit * CT + t) * dkp + i, true);
        }
    };
    fetch(c0, 0);
    for (int c = c0; c < c1; ++c) {
        const size_t unit = (size_t)c * p.H + h;
        const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, stage = stages == 2 ? (c - c0) & 1 : 0;
        const float* w = smem + stage * walk_stage(dkp);
        const float* k = w + CT * wp;
        copies_done();
        __syncthreads();
        if (stages == 2 && c + 1 < c1) fetch(c + 1, stage ^ 1);
        if (n <= 0 || n > CT) {                         // token by token: sixteen threads share a column
            const int col = tid >> 4, part = tid & 15, hq = h / p.group;
            for (int t = t0; t < t0 + n; ++t) {
                const float* kr = p.k + (size_t)t * p.ldk + hq * p.dk;
                const float* qr = p.q + (size_t)t * p.ldq + hq * p.dk;
                const float* gr = p.g + (size_t)t * p.ldg + h * p.dk;
                float held = 0.f, o = 0.f;
                for (int i = part; i < p.dk; i += 16) {
                    sS[i * WC + col] *= gr[i];
                    held = fmaf(sS[i * WC + col], kr[i], held);
                }
                for (int x = 8; x > 0; x >>= 1) held += __shfl_xor_sync(0xffffffffu, held, x);
                const float v = col < n_cols ? p.v[(size_t)t * p.ldv + (size_t)h * p.dv + col0 + col] : 0.f;
                const float u = p.beta[(size_t)t * p.ldb + h] * (v - held);
                for (int i = part; i < p.dk; i += 16) {
                    const float now = fmaf(kr[i], u, sS[i * WC + col]);
                    sS[i * WC + col] = now;
                    o = fmaf(now, qr[i], o);
                }
                for (int x = 8; x > 0; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
                if (part == 0 && col < n_cols) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + col0 + col] = o;
            }
            __syncthreads();
            if (stages == 1 && c + 1 < c1) fetch(c + 1, 0);
            continue;
        }
        const int row = tid >> 2, quad = (tid & 3) * 4;  // this thread's four columns of a token's u
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        float* const u_row = p.U + (unit * CT + row) * p.dvp + col0 + quad;
        if (quad < n_cols) u = *reinterpret_cast<const float4*>(u_row);     // rows of dvp: whole pieces of four
        for (int e = tid; e < p.dk * 4; e += WALK) {    // the state this chunk starts from
            const int i = e >> 2, q4 = (e & 3) * 4;
            if (q4 < n_cols)
                *reinterpret_cast<float4*>(p.start + (unit * p.dk + i) * p.dvp + col0 + q4) = *reinterpret_cast<const float4*>(sS + i * WC + q4);
        }
        // W S: a quarter of the channels, four tokens 16 apart and four columns per thread
        {
            const int part = tid >> 6, g = (tid & 63) >> 2, per = (dkp / 4 + 3) / 4 * 4, k1 = min(dkp, (part + 1) * per);
            f32x2 acc[4][2];
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[x][0] = acc[x][1] = 0ull;
#pragma unroll 2
            for (int i = part * per; i < k1; i += 4) {
                float4 a[4];
#pragma unroll
                for (int x = 0; x < 4; ++x) a[x] = *reinterpret_cast<const float4*>(w + (g + 16 * x) * wp + i);
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(sS + (i + y) * WC + quad);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const float v = y == 0 ? a[x].x : y == 1 ? a[x].y : y == 2 ? a[x].z : a[x].w;
                        const f32x2 vv = pack2(v, v);
                        acc[x][0] = fma2(vv, b.x, acc[x][0]);
                        acc[x][1] = fma2(vv, b.y, acc[x][1]);
                    }
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) *reinterpret_cast<ulonglong2*>(red + (part * CT + g + 16 * x) * WC + quad) = make_ulonglong2(acc[x][0], acc[x][1]);
        }
        __syncthreads();
        {
            float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int part = 0; part < 4; ++part) {
                const float4 a = *reinterpret_cast<const float4*>(red + (part * CT + row) * WC + quad);
                sum.x += a.x; sum.y += a.y; sum.z += a.z; sum.w += a.w;
            }
            u.x -= sum.x; u.y -= sum.y; u.z -= sum.z; u.w -= sum.w;
            *reinterpret_cast<float4*>(sU + row * WC + quad) = u;
            if (quad < n_cols) *reinterpret_cast<float4*>(u_row) = u;
        }
        __syncthreads();
        // S <- decay S + K^T u: half of the tokens, four channels and four columns per thread
        const int half = tid >> 7, g = (tid & 127) >> 2;
        for (int base = 0; base < dkp; base += 128) {
            const int i = base + g * 4;
            f32x2 acc[4][2];
#pragma unroll
            for (int x = 0; x < 4; ++x) acc[x][0] = acc[x][1] = 0ull;
            if (i < dkp) {
#pragma unroll 4
                for (int t = half * 32; t < half * 32 + 32; ++t) {
                    const float4 a = *reinterpret_cast<const float4*>(k + t * dkp + i);
                    const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(sU + t * WC + quad);
                    const float f[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
                        const f32x2 aa = pack2(f[x], f[x]);
                        acc[x][0] = fma2(aa, b.x, acc[x][0]);
                        acc[x][1] = fma2(aa, b.y, acc[x][1]);
                    }
                }
                if (half)
#pragma unroll
                    for (int x = 0; x < 4; ++x) *reinterpret_cast<ulonglong2*>(red + (i + x) * WC + quad) = make_ulonglong2(acc[x][0], acc[x][1]);
            }
            __syncthreads();
            if (!half && i < dkp) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const float d = p.decay[unit * dkp + i + x];
                    const float4 more = *reinterpret_cast<const float4*>(red + (i + x) * WC + quad);
                    const float2 a = unpack2(acc[x][0]), b = unpack2(acc[x][1]);
                    float4* at = reinterpret_cast<float4*>(sS + (i + x) * WC + quad);
                    float4 S = *at;
                    S.x = fmaf(d, S.x, a.x + more.x); S.y = fmaf(d, S.y, a.y + more.y); S.z = fmaf(d, S.z, b.x + more.z); S.w = fmaf(d, S.w, b.y + more.w);
                    *at = S;
                }
            }
        }
        if (stages == 1) {
            __syncthreads();
            if (c + 1 < c1) fetch(c + 1, 0);
        }
    }
    __syncthreads();
    for (int e = tid; e < p.dk * WC; e += WALK) {
        const int col = e / p.dk, i = e - col * p.dk;
        if (col < n_cols) own[(size_t)col * p.dk + i] = sS[i * WC + col];
    }
}

constexpr int OS = 32;                                  // key channels of a slice of the outputs' kernel
template <int NC>
constexpr int output_floats() {
    const int stage = OS * CT + 2 * OS * 64 * NC, values = CT * 64 * NC;
    return (stage > values ? stage : values) + CT * PP;
}

template <int NC>
__global__ void __launch_bounds__(THREADS, 3)
delta_output_kernel(Delta p) {
    constexpr int COLS = 64 * NC, FOURS = OS / 4, NQ = CT * FOURS / THREADS, NV = CT * 16 * NC / THREADS;
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                                   // [OS][64 tokens]
    float* ss = sq + OS * CT;                           // two slices [OS][COLS] of the state in turn
    float* svv = smem;                                  // [64 tokens][COLS], after the last slice
    float* sp = smem + output_floats<NC>() - CT * PP;   // [64 j][PP]
    grid_dep_launch();
    grid_dep_wait();
    const int c = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * COLS, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, nv = min(COLS, p.dv - col0);
    if (c == 0)                                         // rows behind the last sequence belong to nobody: a defined value
        for (int r = p.chunk_start[p.n_chunks]; r < p.T_rows; ++r)
            for (int e = tid; e < nv; e += THREADS) p.o[(size_t)r * p.ldo + (size_t)h * p.dv + col0 + e] = 0.f;
    if (n <= 0 || n > CT) return;
    const size_t unit = (size_t)c * p.H + h;
    Raw4<float> rq[NQ];
    auto token_of = [&](int e) { return (e >> 5) * 4 + ((e & 31) >> 3); };
    auto fetch = [&](int i0, float* dst) {
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS;
            get_four(rq[x], p.Q + (unit * CT + token_of(e)) * p.dkp + i0, (e & 7) * 4, p.dkp - i0, true, 1);
        }
#pragma unroll 4
        for (int e = tid; e < OS * 16 * NC; e += THREADS) {
            const int i = e / (16 * NC), col = (e % (16 * NC)) * 4;
            copy16(dst + e * 4, p.start + (unit * p.dk + i0 + i) * p.dvp + col0 + col, i0 + i < p.dk && col < nv);
        }
    };
    fetch(0, ss);
    for (int e = tid; e < CT * 16; e += THREADS)
        *reinterpret_cast<float4*>(sp + (e >> 4) * PP + (e & 15) * 4) = *reinterpret_cast<const float4*>(p.B + unit * CT * CT + e * 4);
    f32x2 acc[8][2 * NC];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 2 * NC; ++j) acc[i][j] = 0ull;
    for (int i0 = 0; i0 < p.dk; i0 += OS) {
        __syncthreads();
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * THREADS, t = token_of(e), i = (e & 7) * 4;
            const float4 a = rq[x].value();
            sq[at_ct(i, t)] = a.x; sq[at_ct(i + 1, t)] = a.y; sq[at_ct(i + 2, t)] = a.z; sq[at_ct(i + 3, t)] = a.w;
        }
        copies_done();
        __syncthreads();
        const float* now = ss + (i0 / OS & 1) * OS * COLS;
        if (i0 + OS < p.dk) fetch(i0 + OS, ss + ((i0 / OS + 1) & 1) * OS * COLS);
        tile_product<NC, true>(acc, sq, now, OS, ty, tx);
    }
    Raw4<float> rv[NV];
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const int e = tid + x * THREADS, j = e / (16 * NC), col = (e % (16 * NC)) * 4;
        get_four(rv[x], p.U + (unit * CT + j) * p.dvp + col0, col, (nv + 3) / 4 * 4, j < n, 1);
    }
    __syncthreads();
    bool odd = false;                                   // a value that is not finite must not meet the weights of zero of earlier tokens
#pragma unroll
    for (int x = 0; x < NV; ++x) {
        const float4 f = rv[x].value();
        odd |= !(fabsf(f.x) <= 3.402823466e38f && fabsf(f.y) <= 3.402823466e38f && fabsf(f.z) <= 3.402823466e38f && fabsf(f.w) <= 3.402823466e38f);
        *reinterpret_cast<float4*>(svv + (tid + x * THREADS) * 4) = f;
    }
    odd = __syncthreads_or(odd);
    if (odd) add_values<NC, 1, true>(acc, sp, svv, n, ty, tx);
    else add_values<NC, 1, false>(acc, sp, svv, n, ty, tx);
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int t = (i >> 2) * 32 + ty * 4 + (i & 3);
        if (t >= n) continue;
#pragma unroll
        for (int g = 0; g < NC; ++g) {
            const int own = g * 64 + tx * 4;
            float* dst = p.o + (size_t)(t0 + t) * p.ldo + (size_t)h * p.dv + col0 + own;
            const float2 a = unpack2(acc[i][2 * g]), b = unpack2(acc[i][2 * g + 1]);
            if (own < nv) dst[0] = a.x;
            if (own + 1 < nv) dst[1] = a.y;
            if (own + 2 < nv) dst[2] = b.x;
            if (own + 3 < nv) dst[3] = b.y;
        }
    }
}

}  // namespace

// Floats of scratch that `qs_delta_chunks` takes.
QS_API long long qs_delta_chunks_scratch(int n_chunks, int H, int dk, int dv) {
    const long long dkp = (dk + 3) / 4 * 4, dvp = (dv + 3) / 4 * 4;
    return (long long)n_chunks * H * (CT * (3 * dkp + dvp + CT) + dkp + dk * dvp);
}

// q, k [T, (H / group) dk], v [T, H dv], g [T, H dk] (decays), beta [T, H], all float32; o [T, H dv]; state float32 [slots][H][dv][dk].
QS_API int qs_delta_chunks(float* o, long long ldo, const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv, const float* g,
                           long long ldg, const float* beta, long long ldb, float* state, long long slot_stride, const int32_t* seq_slot, int n_seq, int T_rows,
                           int H, int group, int dk, int dv, const int32_t* chunk_start, int n_chunks, const int32_t* seq_chunk, float* scratch,
                           cudaStream_t stream) {
    if (n_seq == 0 || T_rows == 0) return QS_OK;
    QS_REQUIRE(n_seq > 0 && T_rows > 0 && H > 0 && dk > 0 && dv > 0 && n_chunks > 0 && group > 0 && H % group == 0, "delta_chunks: bad sizes");
    QS_REQUIRE(dk <= 256 && H <= 65535 && (dv + WC - 1) / WC <= 65535, "delta_chunks: %d key channels per head above 256", dk);
    QS_REQUIRE(((uintptr_t)scratch % 16) == 0, "delta_chunks: scratch must be 16-byte aligned");
    auto fours = [&](const float* ptr, long long ld) { return (int)(dk % 4 == 0 && ld % 4 == 0 && ((uintptr_t)ptr % 16) == 0); };
    Delta p = {};
    p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.ldq = (size_t)ldq; p.ldk = (size_t)ldk; p.ldv = (size_t)ldv; p.ldg = (size_t)ldg; p.ldb = (size_t)ldb;
    p.chunk_start = chunk_start; p.seq_chunk = seq_chunk; p.seq_slot = seq_slot; p.state = state; p.slot_stride = (size_t)slot_stride;
    p.o = o; p.ldo = (size_t)ldo; p.H = H; p.dk = dk; p.dv = dv; p.dkp = (dk + 3) / 4 * 4; p.dvp = (dv + 3) / 4 * 4; p.group = group;
    p.n_chunks = n_chunks; p.T_rows = T_rows; p.vec_q = fours(q, ldq); p.vec_k = fours(k, ldk); p.vec_g = fours(g, ldg);
    const size_t units = (size_t)n_chunks * H;
    p.W = scratch;
    p.K = p.W + units * CT * p.dkp;
    p.Q = p.K + units * CT * p.dkp;
    p.U = p.Q + units * CT * p.dkp;
    p.B = p.U + units * CT * p.dvp;
    p.decay = p.B + units * CT * CT;
    p.start = p.decay + units * p.dkp;
    cudaError_t e = cudaFuncSetAttribute(delta_terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TERMS_SMEM);
    if (e == cudaSuccess) e = qs_launch_dependent(delta_terms_kernel, dim3(n_chunks, H), dim3(THREADS), TERMS_SMEM, stream, p);
    const size_t walk = walk_smem(p.dkp);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk);
    if (e == cudaSuccess) e = qs_launch_dependent(delta_walk_kernel, dim3(n_seq, H, (dv + WC - 1) / WC), dim3(WALK), walk, stream, p, walk_stages(p.dkp));
#define GO(NC) do { const size_t smem = output_floats<NC>() * sizeof(float); \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_output_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e == cudaSuccess) e = qs_launch_dependent(delta_output_kernel<NC>, dim3(n_chunks, H, (dv + 64 * NC - 1) / (64 * NC)), dim3(THREADS), smem, stream, p); } while (0)
    if (dv > 64) GO(2); else GO(1);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "delta_chunks: %s", cudaGetErrorString(e));
    return qs_check_launch("delta_chunks");
}
