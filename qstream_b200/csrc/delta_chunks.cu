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
// 32-bit numbers and sums throughout, products on the tensor cores as exact products of bfloat16 terms (terms.cuh); decays only as products of factors up to one.  Three walks of every chunk token by token (what it does to an
// identity, what it writes from nothing, its outputs) and a product of dk x dk matrices in the prefix stood here before: 2,000 tokens, 16
// heads of 128 x 128, with their projections, convolutions and norms 1,678 us, now 381 (the terms 108, the walk 118, the outputs 30).
#include "scan.cuh"
#include "scan_tiles.cuh"
#include "term_tiles.cuh"

namespace {

constexpr int WC = 16;                                  // value columns of a block of the walk
constexpr int WALK = 256;

struct Delta {
    const float *q, *k, *v, *g, *beta;                  // rows of ldq, ldk, ldv, ldg, ldb
    size_t ldq, ldk, ldv, ldg, ldb;
    const int32_t *chunk_start, *seq_chunk, *seq_slot;
    float *W, *K, *Q;                                   // [chunks][H][64][dkp]: the solution's W, k times the decays behind it, q times those before
    __nv_bfloat16 *K3;                                  // up to 128 channels, instead of K: its terms [chunks][H][3][64][dk8]
    float *U;                                           // [chunks][H][64][dvp]
    float *B;                                           // [chunks][H][64 j][64 t]
    float *decay;                                       // [chunks][H][dkp]
    float *start;                                       // [chunks][H][dk][dvp]: the states the chunks start from
    float *state; size_t slot_stride;
    float *o; size_t ldo;
    int H, dk, dv, dkp, dvp, dk8, group, n_chunks, T_rows;
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

// TERM_PLANES: K goes on as terms, split once instead of by every block of the walk (W as terms too: six 2-byte stores for two 4-byte ones in
// the unrolled substitution, 130 us instead of 108).
template <bool TERM_PLANES>
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
        if (i0 + i < (TERM_PLANES ? p.dk8 : p.dkp)) {  // zeros from dk on
            float e0[4], e1[4], e2[4], e3[4];
#pragma unroll
            for (int y = 0; y < 4; ++y) {
                e0[y] = edge[i + y];
                e1[y] = e0[y] * edge[PASS + i + y];
                e2[y] = e1[y] * edge[2 * PASS + i + y];
                e3[y] = edge[3 * PASS + i + y];
            }
            const bool in = !TERM_PLANES || i0 + i < p.dkp;
            if (second && lane < 8 && in)
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
                if (in) {
                    *reinterpret_cast<float4*>(p.Q + at) = make_float4(q[0], q[1], q[2], q[3]);
                    *reinterpret_cast<float4*>(p.W + at) = make_float4(w[0], w[1], w[2], w[3]);
                }
                if (TERM_PLANES) {
                    uint32_t a[3], b[3];
                    terms_of(pack2(k[0], k[1]), a[0], a[1], a[2]);
                    terms_of(pack2(k[2], k[3]), b[0], b[1], b[2]);
#pragma unroll
                    for (int x = 0; x < 3; ++x)
                        *reinterpret_cast<uint2*>(p.K3 + ((unit * 3 + x) * CT + t) * p.dk8 + i0 + i) = make_uint2(a[x], b[x]);
                } else *reinterpret_cast<float4*>(p.K + at) = make_float4(k[0], k[1], k[2], k[3]);
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
inline size_t walk_smem(int dkp) {
    return (size_t)(walk_stage(dkp) + dkp * WC + CT * WC + (4 * CT * WC > dkp * WC ? 4 * CT * WC : dkp * WC)) * sizeof(float);
}

// The walk for more than 128 key channels, by multiply-adds.  Two blocks to an SM in the bounds, as many as shared memory holds: left to
// itself the compiler took 80 registers and spilled, 4,000 tokens of 8 heads of 256 x 128 536 us instead of 466.
__global__ void __launch_bounds__(WALK, 2)
delta_walk_kernel(Delta p) {
    extern __shared__ __align__(16) float smem[];
    const int dkp = p.dkp, wp = dkp + 4;
    float* sS = smem + walk_stage(dkp);                 // [dk][16]
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
    auto fetch = [&](int c) {
        const int n = p.chunk_start[c + 1] - p.chunk_start[c];
        if (n <= 0 || n > CT) return;
        const size_t unit = (size_t)c * p.H + h;
        float* w = smem;
        float* k = w + CT * wp;
        const int fours = dkp / 4;
        for (int e = tid; e < CT * fours; e += WALK) {
            const int t = e / fours, i = (e - t * fours) * 4;
            copy16(w + t * wp + i, p.W + (unit * CT + t) * dkp + i, true);
            copy16(k + t * dkp + i, p.K + (unit * CT + t) * dkp + i, true);
        }
    };
    fetch(c0);
    for (int c = c0; c < c1; ++c) {
        const size_t unit = (size_t)c * p.H + h;
        const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0;
        const float* w = smem;
        const float* k = w + CT * wp;
        copies_done();
        __syncthreads();
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
            if (c + 1 < c1) fetch(c + 1);
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
            if (row >= n) u = make_float4(0.f, 0.f, 0.f, 0.f);      // nobody's token writes nothing, whatever the state holds
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
        __syncthreads();
        if (c + 1 < c1) fetch(c + 1);
    }
    __syncthreads();
    for (int e = tid; e < p.dk * WC; e += WALK) {
        const int col = e / p.dk, i = e - col * p.dk;
        if (col < n_cols) own[(size_t)col * p.dk + i] = sS[i * WC + col];
    }
}

// The walk for up to 128 key channels, on the tensor cores (mma.sync, three bfloat16 terms per number, terms.cuh): a block holds 16 value columns of
// one head's state, each of its eight warps 16 channels of it in registers; the state's terms, u's and those of W and K lie in shared memory.
//   1  W S: a warp takes 16 tokens and half of the channels; the halves meet in shared memory, u = U - W S, as terms
//   2  S <- decay S + K^T u: a warp's 16 channels over all 64 tokens; the state's terms
// W of the next chunk becomes terms while u is formed (the one after that is on its way in registers), K is copied in behind the second
// step, as terms that the kernel before has split.
//
// A chain of 32 steps for 2,000 tokens of 16 heads of 128 x 128.  By multiply-adds a step took 4.2 us (shared memory's pipe: eight 16-byte reads per 32 paired
// multiply-adds), 133 us in all; with each block splitting W and K for itself 119; now
// 113; with the way back for sums whose operands the terms do not hold (calls that no ordinary step makes) 118.  With sixteen warps, each half of
// the columns: 119 instead of 113 (64 channels: 4 us less of 73).
// MC channels, 64 or 128; pitches of W and K, of S and u: rows of 16 bytes meet all banks
constexpr int SP = WC + 8;
template <int MC> constexpr int mma_walk_smem() { return (2 * 3 * CT * (MC + 8) + 3 * MC * SP + 3 * CT * SP) * 2 + CT * WC * 4; }

__device__ __forceinline__ void put_four(__nv_bfloat16* at, int term, float4 f) {
    uint32_t a[3], b[3];
    terms_of(pack2(f.x, f.y), a[0], a[1], a[2]);
    terms_of(pack2(f.z, f.w), b[0], b[1], b[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint2*>(at + i * term) = make_uint2(a[i], b[i]);
}
__device__ __forceinline__ void put_two(__nv_bfloat16* at, int term, float x, float y) {
    uint32_t a[3];
    terms_of(pack2(x, y), a[0], a[1], a[2]);
#pragma unroll
    for (int i = 0; i < 3; ++i) *reinterpret_cast<uint32_t*>(at + i * term) = a[i];
}

// The sums of the walk whose operands the terms did not hold, by multiply-adds: token t's W S, and channel i of the state after chunk c.
__device__ __noinline__ float plain_held(const Delta& p, size_t unit, int t, int col) {
    const float *w = p.W + (unit * CT + t) * p.dkp, *S = p.start + unit * p.dk * p.dvp + col;
    float sum = 0.f;
    for (int i = 0; i < p.dk && sum == sum; ++i) sum = fmaf(w[i], S[(size_t)i * p.dvp], sum);        // NaN stays NaN
    return sum;
}
__device__ __noinline__ float plain_state(const Delta& p, int c, int h, int i, int col) {
    const size_t unit = (size_t)c * p.H + h;
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0;
    float sum = 0.f, run = 1.f;
    for (int t = n - 1; t >= 0 && sum == sum; --t) {
        sum = fmaf(p.k[(size_t)(t0 + t) * p.ldk + h / p.group * p.dk + i] * run, p.U[(unit * CT + t) * p.dvp + col], sum);
        run *= p.g[(size_t)(t0 + t) * p.ldg + h * p.dk + i];
    }
    return fmaf(p.decay[unit * p.dkp + i], p.start[(unit * p.dk + i) * p.dvp + col], sum);
}

template <int MC>
__global__ void __launch_bounds__(2 * MC)
delta_walk_mma_kernel(const __grid_constant__ Delta p) {
    constexpr int MP = MC + 8, WALKERS = 2 * MC, PARTS = MC / 64;
    extern __shared__ __align__(16) float smem[];
    __nv_bfloat16* const tw = reinterpret_cast<__nv_bfloat16*>(smem);      // [3][64 tokens][MP]
    __nv_bfloat16* const tk = tw + 3 * CT * MP;
    __nv_bfloat16* const ts = tk + 3 * CT * MP;         // [3][MC channels][SP]
    __nv_bfloat16* const tu = ts + 3 * MC * SP;         // [3][64 tokens][SP]
    float* const red = reinterpret_cast<float*>(tu + 3 * CT * SP);         // [64][16]
    grid_dep_launch();
    grid_dep_wait();
    const int s = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * WC, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q2 = (lane & 3) * 2;
    const int slot = p.seq_slot[s], c0 = p.seq_chunk[s], c1 = p.seq_chunk[s + 1], dkp = p.dkp;
    if (slot < 0 || c1 <= c0) return;
    const int n_cols = min(WC, p.dv - col0);
    float* own = p.state + (size_t)slot * p.slot_stride + ((size_t)h * p.dv + col0) * p.dk;
    // the warp's channels warp 16 + g and + 8, columns 8 y + q2 and + 1
    float S[2][2][2];
    auto each = [&](auto f) {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y)
#pragma unroll
                for (int z = 0; z < 2; ++z) f(S[x][y][z], warp * 16 + 8 * x + g, 8 * y + q2 + z);
    };
    auto put_state = [&]() {
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) put_two(ts + (warp * 16 + 8 * x + g) * SP + 8 * y + q2, MC * SP, S[x][y][0], S[x][y][1]);
    };
    each([&](float& v, int i, int col) { v = i < p.dk && col < n_cols ? own[(size_t)col * p.dk + i] : 0.f; });
    put_state();
    // W of a chunk on its way to registers, and as terms to shared memory; the terms of K on their way there (columns behind dk8 stay zeros)
    constexpr int ROW = MC / 4, PIECES = CT * ROW / WALKERS;
    float4 rw[PIECES];
    auto whole = [&](int c) {
        const int n = c < c1 ? p.chunk_start[c + 1] - p.chunk_start[c] : 0;
        return n > 0 && n <= CT;
    };
    // The state after chunk c, where the terms did not hold what chunk c wrote.  Looked at where a chunk's u shows it (what is no number makes all u of its
    // column none, what is small counts only where they are) and at the end.
    auto mend_state = [&](int c) {
        if (c < c0 || !whole(c)) return;
        each([&](float& v, int i, int col) { if (!held(v) && i < p.dk && col < n_cols) v = plain_state(p, c, h, i, col0 + col); });
    };
    const int w_at = tid / ROW, w_i = tid % ROW * 4;
    auto fetch_w = [&](int c) {
        const bool have = whole(c) && w_i < dkp;
        const float* from = p.W + (((size_t)c * p.H + h) * CT + w_at) * dkp + w_i;
#pragma unroll
        for (int x = 0; x < PIECES; ++x) rw[x] = have ? *reinterpret_cast<const float4*>(from + x * (WALKERS / ROW) * dkp) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto put_w = [&]() {
#pragma unroll
        for (int x = 0; x < PIECES; ++x) put_four(tw + (w_at + x * (WALKERS / ROW)) * MP + w_i, CT * MP, rw[x]);
    };
    constexpr int KROW = MC / 8;
    const int k_at = tid / KROW, k_i = tid % KROW * 8;
    const uint32_t k_to = (uint32_t)__cvta_generic_to_shared(tk) + (k_at * MP + k_i) * 2;
    auto copy_k = [&](int c) {
        if (whole(c) && k_i < p.dk8) {
            const __nv_bfloat16* from = p.K3 + (((size_t)c * p.H + h) * 3 * CT + k_at) * p.dk8 + k_i;
#pragma unroll
            for (int x = 0; x < 3 * CT * KROW / WALKERS; ++x)
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(k_to + x * (WALKERS / KROW) * MP * 2), "l"(from + x * (WALKERS / KROW) * p.dk8) : "memory");
        }
    };
    if (p.dk8 < MC) {
        for (int e = tid; e < 3 * CT * MP / 2; e += WALKERS) reinterpret_cast<uint32_t*>(tk)[e] = 0u;
        __syncthreads();
    }
    fetch_w(c0);
    copy_k(c0);
    put_w();
    fetch_w(c0 + 1);
    copies_done();
    const uint32_t aw = (uint32_t)__cvta_generic_to_shared(tw), ak = (uint32_t)__cvta_generic_to_shared(tk);
    const uint32_t as = (uint32_t)__cvta_generic_to_shared(ts), au = (uint32_t)__cvta_generic_to_shared(tu);
    __syncthreads();
    for (int c = c0; c < c1; ++c) {
        const size_t unit = (size_t)c * p.H + h;
        const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0;
        if (n <= 0 || n > CT) {                         // token by token on the state in 32-bit, over u's and the state's terms: sixteen threads share a column
            mend_state(c - 1);
            float* sS = reinterpret_cast<float*>(ts);   // [MC][17]
            each([&](float& v, int i, int col) { if (i < p.dk) sS[i * 17 + col] = v; });
            __syncthreads();
            const int hq = h / p.group, part = tid & 15;
            for (int col = tid >> 4; col < WC; col += WALKERS / 16)
                for (int t = t0; t < t0 + n; ++t) {
                    const float* kr = p.k + (size_t)t * p.ldk + hq * p.dk;
                    const float* qr = p.q + (size_t)t * p.ldq + hq * p.dk;
                    const float* gr = p.g + (size_t)t * p.ldg + h * p.dk;
                    float held = 0.f, o = 0.f;
                    for (int i = part; i < p.dk; i += 16) {
                        sS[i * 17 + col] *= gr[i];
                        held = fmaf(sS[i * 17 + col], kr[i], held);
                    }
                    for (int x = 8; x > 0; x >>= 1) held += __shfl_xor_sync(0xffffffffu, held, x);
                    const float v = col < n_cols ? p.v[(size_t)t * p.ldv + (size_t)h * p.dv + col0 + col] : 0.f;
                    const float u = p.beta[(size_t)t * p.ldb + h] * (v - held);
                    for (int i = part; i < p.dk; i += 16) {
                        const float now = fmaf(kr[i], u, sS[i * 17 + col]);
                        sS[i * 17 + col] = now;
                        o = fmaf(now, qr[i], o);
                    }
                    for (int x = 8; x > 0; x >>= 1) o += __shfl_xor_sync(0xffffffffu, o, x);
                    if (part == 0 && col < n_cols) p.o[(size_t)t * p.ldo + (size_t)h * p.dv + col0 + col] = o;
                }
            __syncthreads();
            each([&](float& v, int i, int at) { v = i < p.dk ? sS[i * 17 + at] : 0.f; });
            __syncthreads();
            put_state();
            put_w();
            fetch_w(c + 2);
            copy_k(c + 1);
            copies_done();
            __syncthreads();
            continue;
        }
        // 1
        const int tile = warp & 3, part = warp >> 2;
        float y[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}}, u[2][2][2];
        if (part == 0)                                  // what the tokens write from nothing
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const float2 two = 8 * z + q2 < n_cols ? *reinterpret_cast<const float2*>(p.U + (unit * CT + tile * 16 + 8 * x + g) * p.dvp + col0 + 8 * z + q2)
                                                           : make_float2(0.f, 0.f);
                    u[x][z][0] = two.x;
                    u[x][z][1] = two.y;
                }
        float d[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int i = warp * 16 + 8 * x + g;
            d[x] = i < dkp ? p.decay[unit * dkp + i] : 0.f;
        }
        auto put_start = [&]() {                        // the state this chunk starts from
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const int i = warp * 16 + 8 * x + g, col = 8 * z + q2;
                    if (i < p.dk && col < n_cols) *reinterpret_cast<float2*>(p.start + (unit * p.dk + i) * p.dvp + col0 + col) = make_float2(S[x][z][0], S[x][z][1]);
                }
        };
        put_start();
#pragma unroll
        for (int i = part * 64; i < part * 64 + 64; i += 16) {
            uint32_t a[3][4], b[3][4];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                load_matrices(a[x], aw + x * CT * MP * 2 + rows_first(tile * 16, i, MP, lane));
                load_matrices_turned(b[x], as + x * MC * SP * 2 + rows_first(i, 0, SP, lane));
            }
            add_product<3, 3>(y[0], a, b, 0);
            add_product<3, 3>(y[1], a, b, 1);
        }
        if (PARTS > 1 && part)
#pragma unroll
            for (int z = 0; z < 2; ++z)
#pragma unroll
                for (int x = 0; x < 2; ++x) *reinterpret_cast<float2*>(red + (tile * 16 + 8 * x + g) * WC + 8 * z + q2) = make_float2(y[z][2 * x], y[z][2 * x + 1]);
        __syncthreads();
        uint32_t odd = 0;
        const int tg = tile * 16 + g;
        auto put_u = [&]() {
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const int t = tg + 8 * x, col = 8 * z + q2;
                    put_two(tu + t * SP + col, CT * SP, y[z][2 * x], y[z][2 * x + 1]);
                    if (col < n_cols) *reinterpret_cast<float2*>(p.U + (unit * CT + t) * p.dvp + col0 + col) = make_float2(y[z][2 * x], y[z][2 * x + 1]);
                }
        };
        if (part == 0) {
#pragma unroll
            for (int x = 0; x < 2; ++x)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const float2 more = PARTS > 1 ? *reinterpret_cast<const float2*>(red + (tg + 8 * x) * WC + 8 * z + q2) : make_float2(0.f, 0.f);
                    const bool have = tg + 8 * x < n;   // nobody's tokens write nothing, whatever the state holds
                    y[z][2 * x] = have ? u[x][z][0] - (y[z][2 * x] + more.x) : 0.f;
                    y[z][2 * x + 1] = have ? u[x][z][1] - (y[z][2 * x + 1] + more.y) : 0.f;
                    if (have) odd = max(odd, max(beyond(y[z][2 * x]), beyond(y[z][2 * x + 1])));
                }
            put_u();
        }
        put_w();                                        // behind the barrier: nobody reads W any more
        fetch_w(c + 2);
        copies_done();                                  // this chunk's K
        if (__syncthreads_or(odd > HELD)) {             // u whose operands the terms did not hold
            mend_state(c - 1);
            put_start();
            __syncthreads();
            if (odd > HELD) {
#pragma unroll
                for (int x = 0; x < 2; ++x)
#pragma unroll
                    for (int z = 0; z < 2; ++z)
#pragma unroll
                        for (int e = 0; e < 2; ++e) {
                            const int t = tg + 8 * x, col = 8 * z + q2 + e;
                            if (t < n && !held(y[z][2 * x + e]) && col < n_cols) y[z][2 * x + e] = u[x][z][e] - plain_held(p, unit, t, col0 + col);
                        }
                put_u();
            }
            __syncthreads();
        }
        // 2
        float more[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
        for (int t = 0; t < CT; t += 16) {
            uint32_t a[3][4], b[3][4];
#pragma unroll
            for (int x = 0; x < 3; ++x) {
                load_matrices_turned(a[x], ak + x * CT * MP * 2 + columns_first(t, warp * 16, MP, lane));
                load_matrices_turned(b[x], au + x * CT * SP * 2 + rows_first(t, 0, SP, lane));
            }
            add_product<3, 3>(more[0], a, b, 0);
            add_product<3, 3>(more[1], a, b, 1);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int z = 0; z < 2; ++z)
#pragma unroll
                for (int e = 0; e < 2; ++e) S[x][z][e] = fmaf(d[x], S[x][z][e], more[z][2 * x + e]);
        put_state();
        __syncthreads();
        copy_k(c + 1);
    }
    uint32_t odd_state = 0;
    each([&](float& v, int, int) { odd_state = max(odd_state, beyond(v)); });
    if (odd_state > HELD) mend_state(c1 - 1);
    each([&](float& v, int i, int col) { if (i < p.dk && col < n_cols) own[(size_t)col * p.dk + i] = v; });
}

// The outputs on tcgen05, three terms per number: a block takes a chunk's 64 tokens and 128 value columns (on the TMEM lanes, so that a warp stores 32
// neighbouring ones).  Slices of 64 channels are runs in the unit, summed up in registers; then the weights against u.
constexpr int OUT_THREADS = 256, OUT_SMEM = 1024 + 9 * TILE;
// MANY: more than 128 channels, more than two runs.
template <bool MANY>
__global__ void __launch_bounds__(OUT_THREADS, 2)
delta_output_kernel(const __grid_constant__ Delta p, int32_t* __restrict__ status) {
    constexpr int NQ = CT * 16 / OUT_THREADS, NS = 2 * NQ;
    constexpr uint32_t TMEM = 128;                      // two runs' sums [128 columns][64 tokens]
    extern __shared__ uint8_t smem_raw[];
    __shared__ uint64_t done;
    __shared__ uint32_t tmem_slot;
    const int c = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * 128, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, quad = warp & 3, half = warp >> 2;
    if (tid == 0) { mbar_init(&done, 1); mbar_fence_init(); }
    if (warp == 0) { tmem_alloc(&tmem_slot, TMEM); tmem_relinquish(); }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    grid_dep_launch();
    grid_dep_wait();
    const uint32_t tmem = tmem_slot, own = tmem + ((uint32_t)(quad * 32) << 16) + half * 32;
    const uint32_t tq = (smem_u32(smem_raw) + 1023) & ~1023u, ts = tq + 3 * TILE;       // [3][tokens], [3][2 halves of the columns][channels]
    const uint32_t tb = tq, tu = tb + 3 * TILE;         // after the slices: the weights [3][earlier tokens], u [3][2][tokens]
    const int t0 = p.chunk_start[c], n = p.chunk_start[c + 1] - t0, nv = min(128, p.dv - col0);
    const size_t unit = (size_t)c * p.H + h;
    auto leave = [&]() {
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0) tmem_dealloc(tmem, TMEM);
    };
    if (c == 0)                                         // rows behind the last sequence belong to nobody: a defined value
        for (int r = p.chunk_start[p.n_chunks]; r < p.T_rows; ++r)
            for (int e = tid; e < nv; e += OUT_THREADS) p.o[(size_t)r * p.ldo + (size_t)h * p.dv + col0 + e] = 0.f;
    if (n <= 0 || n > CT) { leave(); return; }
    const int slices = (p.dk + 63) / 64;
    float out[32];
    bool ok = true;
    for (int s = 0; s < slices; ++s) {
        const int i0 = s * 64;
        float4 rq[NQ], rs[NS];
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * OUT_THREADS, i = i0 + (e & 15) * 4;
            rq[x] = i < p.dkp ? *reinterpret_cast<const float4*>(p.Q + (unit * CT + (e >> 4)) * p.dkp + i) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * OUT_THREADS, i = i0 + (e >> 5), col = col0 + (e & 31) * 4;
            rs[x] = i < p.dk && col < p.dvp ? *reinterpret_cast<const float4*>(p.start + (unit * p.dk + i) * p.dvp + col) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        if (s && ok) ok = wait_done(&done, (s - 1) & 1, status);
        if (MANY && s >= 2) {
            tc_fence_after_sync();
            take_sums<32>(out, own + (s & 1) * 64, s == 2);
        }
#pragma unroll
        for (int x = 0; x < NQ; ++x) {
            const int e = tid + x * OUT_THREADS;
            put_terms<3>(tq + place_in_tile(e >> 4, (e & 15) * 4), TILE, rq[x]);
        }
#pragma unroll
        for (int x = 0; x < NS; ++x) {
            const int e = tid + x * OUT_THREADS, col = (e & 31) * 4;
            put_terms<3>(ts + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, rs[x]);
        }
        fence_proxy_async_smem();
        tc_fence_before_sync();
        __syncthreads();
        if (warp == 0 && elect_one()) {
            tc_fence_after_sync();
            multiply_tiles<3, 3, true, false>(tmem + (s & 1) * 64, ts, 2 * TILE, tq, TILE, CT);       // S0^T Q
            mma_commit(&done);
        }
        __syncwarp();
    }
    float4 rb[NQ], ru[NS];
#pragma unroll
    for (int x = 0; x < NQ; ++x) rb[x] = *reinterpret_cast<const float4*>(p.B + unit * CT * CT + (tid + x * OUT_THREADS) * 4);
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * OUT_THREADS, j = e >> 5, col = col0 + (e & 31) * 4;
        ru[x] = j < n && col < p.dvp ? *reinterpret_cast<const float4*>(p.U + (unit * CT + j) * p.dvp + col) : make_float4(0.f, 0.f, 0.f, 0.f);
    }
    if (ok) ok = wait_done(&done, (slices - 1) & 1, status);
    tc_fence_after_sync();
#pragma unroll
    for (int x = 0; x < NQ; ++x) {
        const int e = tid + x * OUT_THREADS;
        put_terms<3>(tb + place_in_tile(e >> 4, (e & 15) * 4), TILE, rb[x]);
    }
#pragma unroll
    for (int x = 0; x < NS; ++x) {
        const int e = tid + x * OUT_THREADS, col = (e & 31) * 4;
        put_terms<3>(tu + (col >> 6) * TILE + place_in_tile(e >> 5, col & 63), 2 * TILE, ru[x]);
    }
    const int older = slices & 1, newer = older ^ 1;
    if (slices > 1) take_sums<32>(out, own + older * 64, slices == 2);
    take_sums<32>(out, own + newer * 64, slices == 1);
    fence_proxy_async_smem();
    tc_fence_before_sync();
    __syncthreads();
    if (warp == 0 && elect_one()) {
        tc_fence_after_sync();
        multiply_tiles<3, 3, true, true>(tmem, tu, 2 * TILE, tb, TILE, CT);       // u^T B
        mma_commit(&done);
    }
    __syncwarp();
    if (ok) ok = wait_done(&done, slices & 1, status);
    tc_fence_after_sync();
    take_sums<32>(out, own, false);
    const int in = quad * 32 + lane, rows = n - half * 32;
    if (in < nv) {
        float* o = p.o + (size_t)t0 * p.ldo + (size_t)h * p.dv + col0 + in;
        uint32_t odd = 0;
#pragma unroll
        for (int x = 0; x < 32; ++x) {
            odd = max(odd, beyond(out[x]));
            if (x < rows) o[(size_t)(half * 32 + x) * p.ldo] = out[x];
        }
        if (odd > HELD)                                 // by multiply-adds, where the terms did not hold the operands: a later token's u meets no earlier one
            for (int t = half * 32; t < min(n, half * 32 + 32); ++t) {
                float v = o[(size_t)t * p.ldo];
                if (held(v)) continue;
                v = 0.f;
                for (int i = 0; i < p.dk && v == v; ++i) v = fmaf(p.Q[(unit * CT + t) * p.dkp + i], p.start[(unit * p.dk + i) * p.dvp + col0 + in], v);
                for (int j = 0; j <= t && v == v; ++j) v = fmaf(p.B[unit * CT * CT + j * CT + t], p.U[(unit * CT + j) * p.dvp + col0 + in], v);
                o[(size_t)t * p.ldo] = v;
            }
    }
    leave();
}

}  // namespace

// Floats of scratch that `qs_delta_chunks` takes.
QS_API long long qs_delta_chunks_scratch(int n_chunks, int H, int dk, int dv) {
    const long long dkp = (dk + 3) / 4 * 4, dvp = (dv + 3) / 4 * 4;
    const long long k_or_terms = dk <= 128 ? (3 * ((dk + 7) / 8 * 8) + 1) / 2 : dkp;       // K, or its terms
    return (long long)n_chunks * H * (CT * (2 * dkp + k_or_terms + dvp + CT) + dkp + dk * dvp);
}

// q, k [T, (H / group) dk], v [T, H dv], g [T, H dk] (decays), beta [T, H], all float32; o [T, H dv]; state float32 [slots][H][dv][dk].
QS_API int qs_delta_chunks(float* o, long long ldo, const float* q, long long ldq, const float* k, long long ldk, const float* v, long long ldv, const float* g,
                           long long ldg, const float* beta, long long ldb, float* state, long long slot_stride, const int32_t* seq_slot, int n_seq, int T_rows,
                           int H, int group, int dk, int dv, const int32_t* chunk_start, int n_chunks, const int32_t* seq_chunk, float* scratch,
                           int32_t* status, cudaStream_t stream) {
    if (n_seq == 0 || T_rows == 0) return QS_OK;
    QS_REQUIRE(n_seq > 0 && T_rows > 0 && H > 0 && dk > 0 && dv > 0 && n_chunks > 0 && group > 0 && H % group == 0, "delta_chunks: bad sizes");
    QS_REQUIRE(dk <= 256 && H <= 65535 && (dv + WC - 1) / WC <= 65535, "delta_chunks: %d key channels per head above 256", dk);
    QS_REQUIRE(((uintptr_t)scratch % 16) == 0, "delta_chunks: scratch must be 16-byte aligned");
    auto fours = [&](const float* ptr, long long ld) { return (int)(dk % 4 == 0 && ld % 4 == 0 && ((uintptr_t)ptr % 16) == 0); };
    Delta p = {};
    p.q = q; p.k = k; p.v = v; p.g = g; p.beta = beta; p.ldq = (size_t)ldq; p.ldk = (size_t)ldk; p.ldv = (size_t)ldv; p.ldg = (size_t)ldg; p.ldb = (size_t)ldb;
    p.chunk_start = chunk_start; p.seq_chunk = seq_chunk; p.seq_slot = seq_slot; p.state = state; p.slot_stride = (size_t)slot_stride;
    p.o = o; p.ldo = (size_t)ldo; p.H = H; p.dk = dk; p.dv = dv; p.dkp = (dk + 3) / 4 * 4; p.dvp = (dv + 3) / 4 * 4; p.dk8 = (dk + 7) / 8 * 8; p.group = group;
    p.n_chunks = n_chunks; p.T_rows = T_rows; p.vec_q = fours(q, ldq); p.vec_k = fours(k, ldk); p.vec_g = fours(g, ldg);
    const size_t units = (size_t)n_chunks * H;
    p.W = scratch;
    const bool terms = dk <= 128;
    p.K = p.W + units * CT * p.dkp;
    p.K3 = reinterpret_cast<__nv_bfloat16*>(p.K);
    p.Q = p.K + units * CT * (terms ? (3 * p.dk8 + 1) / 2 : p.dkp);
    p.U = p.Q + units * CT * p.dkp;
    p.B = p.U + units * CT * p.dvp;
    p.decay = p.B + units * CT * CT;
    p.start = p.decay + units * p.dkp;
    const auto terms_kernel = terms ? delta_terms_kernel<true> : delta_terms_kernel<false>;
    cudaError_t e = cudaFuncSetAttribute(terms_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TERMS_SMEM);
    if (e == cudaSuccess) e = qs_launch_dependent(terms_kernel, dim3(n_chunks, H), dim3(TERMS), TERMS_SMEM, stream, p);
    const dim3 blocks(n_seq, H, (dv + WC - 1) / WC);
    if (p.dkp <= 64) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_mma_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, mma_walk_smem<64>());
        if (e == cudaSuccess) e = qs_launch_dependent(delta_walk_mma_kernel<64>, blocks, dim3(128), mma_walk_smem<64>(), stream, p);
    } else if (p.dkp <= 128) {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_mma_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, mma_walk_smem<128>());
        if (e == cudaSuccess) e = qs_launch_dependent(delta_walk_mma_kernel<128>, blocks, dim3(256), mma_walk_smem<128>(), stream, p);
    } else {
        if (e == cudaSuccess) e = cudaFuncSetAttribute(delta_walk_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)walk_smem(256));
        if (e == cudaSuccess) e = qs_launch_dependent(delta_walk_kernel, blocks, dim3(WALK), walk_smem(p.dkp), stream, p);
    }
    const auto output = dk > 128 ? delta_output_kernel<true> : delta_output_kernel<false>;
    if (e == cudaSuccess) e = cudaFuncSetAttribute(output, cudaFuncAttributeMaxDynamicSharedMemorySize, OUT_SMEM);
    if (e == cudaSuccess) e = qs_launch_dependent(output, dim3(n_chunks, H, (dv + 127) / 128), dim3(OUT_THREADS), OUT_SMEM, stream, p, status);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "delta_chunks: %s", cudaGetErrorString(e));
    return qs_check_launch("delta_chunks");
}
