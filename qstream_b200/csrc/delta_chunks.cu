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
//                         substitution with a column per thread in registers, the decayed q and k
//   delta_walk_kernel     per sequence, head and 16 value columns, the chunks in order: u and the next state, two small products each
//   delta_output_kernel   per chunk and head, side by side: the outputs
//
// All 32-bit; decays only as products of factors up to one.  Three walks of every chunk token by token (what it does to an
// identity, what it writes from nothing, its outputs) and a product of dk x dk matrices in the prefix stood here before: 2,000 tokens, 16
// heads of 128 x 128, with their projections, convolutions and norms 1,678 us, now 426 (the terms 108, the walk 133, the outputs 56).
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

// The terms.  256 threads in four groups of two warps; a group has 32 of the pass's 128 channels and takes them through all steps by
// itself: inside blocks of 16 tokens the pairs' decays as running products, across blocks as products of q (and k) times the decays
// since their block's start with k times the decays up to that block.  Then the groups' sums are added, and a thread solves for a
// column of W or U, its 64 values in registers.
//
// Bound by instruction issue and shared memory's pipe (a third and four fifths of their rates).  What it took before, 214 us for 2,000 tokens and 16 heads of 128 x 128, was 36,000 instructions per
// warp: a condition and two decays per pair of tokens across blocks, a wait of the whole block between steps, two columns and 2,016
// steps unrolled per thread (more code than the instruction cache holds); now
// 108 us.  128 registers a thread at two blocks per SM; 164 bytes are spilled.
constexpr int TERMS = 256, GROUPS = 4, GCH = 32, PASS = GROUPS * GCH;
constexpr int OWN = 16 * 17;                            // a block's own pairs, [16][17]
constexpr int TERMS_SMEM = (3 * PASS * CT + 4 * PASS) * sizeof(float);
static_assert(GROUPS * (2 * CROSS + 4 * OWN) + CT * CT <= 3 * PASS * CT, "the groups' sums and A lie over the staged channels");
// [channel][64 tokens], pieces of four tokens swapped so that neighbouring channels, and every fourth one, meet different banks
__device__ __forceinline__ int at_pass(int c, int t) { return c * CT + (t ^ (((c ^ (c >> 2)) & 7) << 2)); }
__device__ __forceinline__ void group_wait(int group) { asm volatile("bar.sync %0, 64;" :: "r"(1 + group) : "memory"); }

__global__ void __launch_bounds__(TERMS, 2)
delta_terms_kernel(Delta p) {
    extern __shared__ __align__(16) float smem[];
    float* sq = smem;                                   // [PASS][64 tokens]: q, then q times the decays since its block's start
    float* sk = sq + PASS * CT;                         // k, then k times the decays up to its block's end, the next blocks' starts
    float* sw = sk + PASS * CT;                         // the decays, then k times the decays since its block's start
    float* edge = sw + PASS * CT;                       // [4][PASS] the decays of a block of 16 tokens
    float* sums = smem;                                 // after the passes: [GROUPS][B, A][CROSS], [GROUPS][4 blocks][OWN]
    float* minus = sums + GROUPS * (2 * CROSS + 4 * OWN);       // [64 j][64 t]
    __shared__ float s_beta[CT];
    grid_dep_launch();
    grid_dep_wait();
    const int c = blockIdx.x, h = blockIdx.y, tid = threadIdx.x, lane = tid & 31, group = tid >> 6, second = tid >> 5 & 1;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, hq = h / p.group;
    if (n <= 0 || n > CT) return;                       // longer chunks are walked token by token
    const size_t unit = (size_t)c * p.H + h;
    if (tid < CT) s_beta[tid] = tid < n ? p.beta[(size_t)(t0 + tid) * p.ldb + h] : 0.f;
    const int c0 = group * GCH;                         // the group's channels of a pass
    const int jj = lane & 15, block = second * 2 + (lane >> 4);         // this lane's token within a block
    float da[16], db[16];
    f32x2 x1[2][2], x2[4][2], x3[6][2];
#pragma unroll
    for (int x = 0; x < 16; ++x) da[x] = db[x] = 0.f;
#pragma unroll
    for (int x = 0; x < 6; ++x) {
        if (x < 2) x1[x][0] = x1[x][1] = 0ull;
        if (x < 4) x2[x][0] = x2[x][1] = 0ull;
        x3[x][0] = x3[x][1] = 0ull;
    }
    for (int i0 = 0; i0 < p.dkp; i0 += PASS) {
        const int nk = min(PASS, p.dk - i0), i = c0 + (lane & 7) * 4;
        // eight pieces of four channels by four tokens per step: whole 128-byte lines, and no two lanes of a store on one bank
#pragma unroll
        for (int s = 0; s < 8; s += 4) {
            Raw4<float> rq[4], rk[4], rg[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int t = second * 32 + (s + x) * 4 + (lane >> 3);
                get_four(rq[x], p.q + (size_t)(t0 + t) * p.ldq + hq * p.dk + i0, i, nk, t < n, p.vec_q);
                get_four(rk[x], p.k + (size_t)(t0 + t) * p.ldk + hq * p.dk + i0, i, nk, t < n, p.vec_k);
                get_four(rg[x], p.g + (size_t)(t0 + t) * p.ldg + h * p.dk + i0, i, nk, t < n, p.vec_g);
            }
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const int t = second * 32 + (s + x) * 4 + (lane >> 3);
                const float4 a = rq[x].value(), b = rk[x].value(), d = rg[x].value();
                const float fq[4] = {a.x, a.y, a.z, a.w}, fk[4] = {b.x, b.y, b.z, b.w}, fg[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int at = at_pass(i + y, t);
                    sq[at] = fq[y];
                    sk[at] = fk[y];
                    sw[at] = t < n && i + y < nk ? fg[y] : 1.f;
                }
            }
        }
        group_wait(group);
        // pairs of tokens within a block of 16: lane = token j; where x < j the sums mean nothing
#pragma unroll 1
        for (int e = c0; e < c0 + GCH; ++e) {
            float run = sk[at_pass(e, block * 16 + jj)];
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                const int at = at_pass(e, block * 16 + 4 * b);
                const float4 q4 = *reinterpret_cast<const float4*>(sq + at), k4 = *reinterpret_cast<const float4*>(sk + at);
                const float4 w4 = *reinterpret_cast<const float4*>(sw + at);
                const float fq[4] = {q4.x, q4.y, q4.z, q4.w}, fk[4] = {k4.x, k4.y, k4.z, k4.w}, fw[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const int x = 4 * b + y;
                    if (x > jj) run *= fw[y];
                    da[x] = fmaf(fk[y], run, da[x]);
                    db[x] = fmaf(fq[y], run, db[x]);
                }
            }
        }
        group_wait(group);
        // a lane per channel and half of the tokens: what the decays of a block of 16 do to its tokens
        {
            const int ch = c0 + second * 16 + (lane & 15);
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const int b = (lane >> 4) * 2 + y;
                float4 w[4];
                float run = 1.f;
#pragma unroll
                for (int x = 0; x < 4; ++x) w[x] = *reinterpret_cast<const float4*>(sw + at_pass(ch, b * 16 + 4 * x));
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    const int at = at_pass(ch, b * 16 + 4 * x);
                    float4 q4 = *reinterpret_cast<const float4*>(sq + at), k4 = *reinterpret_cast<const float4*>(sk + at);
                    run *= w[x].x; q4.x *= run; k4.x *= run;
                    run *= w[x].y; q4.y *= run; k4.y *= run;
                    run *= w[x].z; q4.z *= run; k4.z *= run;
                    run *= w[x].w; q4.w *= run; k4.w *= run;
                    *reinterpret_cast<float4*>(sq + at) = q4;
                    *reinterpret_cast<float4*>(sw + at) = k4;
                }
                edge[b * PASS + ch] = run;
                run = 1.f;
#pragma unroll
                for (int x = 3; x >= 0; --x) {
                    const int at = at_pass(ch, b * 16 + 4 * x);
                    float4 k4 = *reinterpret_cast<const float4*>(sk + at);
                    k4.w *= run; run *= w[x].w;
                    k4.z *= run; run *= w[x].z;
                    k4.y *= run; run *= w[x].y;
                    k4.x *= run; run *= w[x].x;
                    *reinterpret_cast<float4*>(sk + at) = k4;
                }
            }
        }
        // a block's tokens against all earlier ones, whose k are taken on to this block's start: one warp for B, the other for A
        const float* X = second ? sw : sq;
        const int ch = c0 + second * 16 + (lane & 15), eighth = (lane >> 4) * 8;
        group_wait(group);
        cross_product<1, GCH, at_pass>(x1, X, sk, c0, lane);
        group_wait(group);
#pragma unroll
        for (int x = 0; x < 2; ++x) scale_four(sk + at_pass(ch, eighth + 4 * x), edge[PASS + ch]);
        group_wait(group);
        cross_product<2, GCH, at_pass>(x2, X, sk, c0, lane);
        group_wait(group);
#pragma unroll
        for (int x = 0; x < 4; ++x) scale_four(sk + at_pass(ch, 2 * eighth + 4 * x), edge[2 * PASS + ch]);
        group_wait(group);
        cross_product<3, GCH, at_pass>(x3, X, sk, c0, lane);
        // relative to the chunk's ends, for the products with the states
        if (i0 + i < p.dkp) {
            float e0[4], e1[4], e2[4], e3[4];
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                e0[y] = edge[i + y];
                e1[y] = e0[y] * edge[PASS + i + y];
                e2[y] = e1[y] * edge[2 * PASS + i + y];
                e3[y] = edge[3 * PASS + i + y];
            }
            if (second && lane < 8)
                *reinterpret_cast<float4*>(p.decay + unit * p.dkp + i0 + i) = make_float4(e2[0] * e3[0], e2[1] * e3[1], e2[2] * e3[2], e2[3] * e3[3]);
#pragma unroll
            for (int s = 0; s < 8; ++s) {
                const int b = second * 2 + (s >> 2), t = second * 32 + s * 4 + (lane >> 3);
                const size_t at = (unit * CT + t) * p.dkp + i0 + i;
                float q[4], w[4], k[4];
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const float before = b == 0 ? 1.f : b == 1 ? e0[y] : b == 2 ? e1[y] : e2[y];
                    const int from = at_pass(i + y, t);
                    q[y] = sq[from] * before;
                    w[y] = sw[from] * before;
                    k[y] = sk[from] * (b == 3 ? 1.f : e3[y]);
                }
                *reinterpret_cast<float4*>(p.Q + at) = make_float4(q[0], q[1], q[2], q[3]);
                *reinterpret_cast<float4*>(p.W + at) = make_float4(w[0], w[1], w[2], w[3]);
                *reinterpret_cast<float4*>(p.K + at) = make_float4(k[0], k[1], k[2], k[3]);
            }
        }
        group_wait(group);
    }
    __syncthreads();
    {
        float* mine = sums + (group * 2 + second) * CROSS;
        cross_store<1>(mine, x1, lane);
        cross_store<2>(mine, x2, lane);
        cross_store<3>(mine, x3, lane);
        float* own = sums + GROUPS * 2 * CROSS + (group * 4 + block) * OWN;     // A at (j, x), x > j; B at (x, j), x >= j
#pragma unroll
        for (int x = 0; x < 16; ++x) {
            if (x > jj) own[jj * 17 + x] = da[x];
            if (x >= jj) own[x * 17 + jj] = db[x];
        }
    }
    __syncthreads();
    for (int e = tid; e < CT * CT; e += TERMS) {
        const int j = e >> 6, t = e & 63, I = t >> 4;
        float a = 0.f, b = 0.f;
        if (I > j >> 4) {
            const float* at = sums + cross_at(I) + (t & 15) * (16 * I + 1) + j;
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) { b += at[g * 2 * CROSS]; a += at[(g * 2 + 1) * CROSS]; }
        } else if (t >= j) {
            const float* at = sums + GROUPS * 2 * CROSS + I * OWN;
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                if (t > j) a += at[g * 4 * OWN + (j & 15) * 17 + (t & 15)];
                b += at[g * 4 * OWN + (t & 15) * 17 + (j & 15)];
            }
        }
        minus[e] = -s_beta[t] * a;
        p.B[unit * CT * CT + e] = b;
    }
    __syncthreads();
    // X[t] = beta_t R[t] - sum_{j < t} beta_t A[t][j] X[j], a column of W (R in place) or U (R: the values) per thread.  A token that is
    // done takes no harm from being "updated" by itself: minus is zero there and nobody reads it any more.
    for (int col = tid; col < p.dk + p.dv; col += TERMS) {
        const bool of_w = col < p.dk;
        const float* from = of_w ? p.W + unit * CT * p.dkp + col : p.v + (size_t)t0 * p.ldv + (size_t)h * p.dv + (col - p.dk);
        const size_t step = of_w ? p.dkp : p.ldv;
        float* to = of_w ? p.W + unit * CT * p.dkp + col : p.U + unit * CT * p.dvp + (col - p.dk);
        const int width = of_w ? p.dkp : p.dvp;
        f32x2 x[CT / 2];
#pragma unroll
        for (int t = 0; t < CT; t += 2)
            x[t / 2] = mul2(pack2(s_beta[t], s_beta[t + 1]), pack2(t < n ? from[t * step] : 0.f, t + 1 < n ? from[(t + 1) * step] : 0.f));
#pragma unroll
        for (int j = 0; j < CT; ++j) {
            const float2 two = unpack2(x[j / 2]);
            const float own = j & 1 ? two.y : two.x;
            to[j * width] = own;
            const f32x2 o = pack2(own, own);
#pragma unroll
            for (int t = (j + 1) / 4 * 4; t < CT; t += 4) {
                const ulonglong2 m = *reinterpret_cast<const ulonglong2*>(minus + j * CT + t);
                x[t / 2] = fma2(m.x, o, x[t / 2]);
                x[t / 2 + 1] = fma2(m.y, o, x[t / 2 + 1]);
            }
        }
    }
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
    if (e == cudaSuccess) e = qs_launch_dependent(delta_terms_kernel, dim3(n_chunks, H), dim3(TERMS), TERMS_SMEM, stream, p);
    const size_t walk = walk_smem(p.dkp);
    // the most any head takes (two stages of 128 channels or one of 256), so that threads with models of other sizes set the same
    const size_t most = walk_smem(256) > walk_smem(128) ? walk_smem(256) : walk_smem(128);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most);
    if (e == cudaSuccess) e = qs_launch_dependent(delta_walk_kernel, dim3(n_seq, H, (dv + WC - 1) / WC), dim3(WALK), walk, stream, p, walk_stages(p.dkp));
#define GO(NC) do { const size_t smem = output_floats<NC>() * sizeof(float); \
    if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_output_kernel<NC>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
    if (e == cudaSuccess) e = qs_launch_dependent(delta_output_kernel<NC>, dim3(n_chunks, H, (dv + 64 * NC - 1) / (64 * NC)), dim3(THREADS), smem, stream, p); } while (0)
    if (dv > 64) GO(2); else GO(1);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "delta_chunks: %s", cudaGetErrorString(e));
    return qs_check_launch("delta_chunks");
}
