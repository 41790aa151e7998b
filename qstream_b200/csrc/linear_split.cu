// C = act(A W^T + bias) + res1 + res2 for float32 A [M, K] and W [N, K] on the 5th-generation tensor cores: every number as
// three bfloat16 terms, six products of terms for one of numbers (terms.cuh).  The unit adds up runs of 64 products, from zero and the small
// terms first; the runs' sums are read back and added in registers with rounded 32-bit additions, in ascending k.  Against float64 that is nearer than the
// CUDA-core product, whose runs of 256 are chains of rounded additions (figures below).
//
// Pairs of CTAs (tcgen05.mma.cta_group::2) work on tiles of 256 features x NT tokens: features on the M side, so that a warp's
// stores are 32 neighbouring features of a token.  Sixteen warps per CTA, each of which does both halves of the work: they fetch the CTA's 128 rows of W and NT / 2 rows of
// A, 64 numbers of each at a time, split them into a stage's six K-major tiles (128-byte swizzle) of a ring, and, one stage
// later, read the run's sums from one of two TMEM accumulators and add them to their own (NT / 4 per thread).  While the unit works on one
// stage the next is split.  A warp more, for the MMAs alone, would leave a thread 96 registers instead of 128: 340 bytes spilled.
//
// Bound by the tensor unit where there are many tiles (2048 x 16384 x 4096: 1,138 us, 240 TFLOP/s of products of 32-bit numbers, six times as
// many in the unit: 0.89 of its measured peak; the CUDA-core product takes 5,155) and else by the chain of a
// k-block: fetch, split, barrier of the pair, MMAs, sums (700 x 6144 x 2048 with K in one part: 96 us, 412 there; leaving out the loads gives 84, the sums'
// way to registers 84, all but barriers, stores and MMAs 82), and by a unit's two ends, where the pipeline fills and drains (9 us at 256 tokens).  Loads four rows of whole 128-byte lines at a time: eight rows of 32 bytes
// per lane took 40 wavefronts instead of 4 each; loads set out as soon as their registers are free: 96 against 102 us
// with all of them behind the barrier; two k-blocks under way for few tokens: no gain, more registers.  Few rows (up to 64 or so) are bound by the latency of that
// chain, W's lines in L2 three k-blocks ahead of the loads (16 x 14336 x 2048 62 -> 57 us; six ahead 59): 64 x 6144 x 2048 35 us (57).
//
// Error against float64, 2-norm, this | CUDA cores, K = 256, 2,048, 8,192: normal numbers 8.7e-8 | 2.9e-7, 1.1e-7 | 2.9e-7, 1.2e-7 | 3.1e-7;
// activations of one sign (squared ReLU) against normal numbers 9.8e-8 | 2.0e-7, 1.2e-7 | 2.1e-7, 1.3e-7 | 2.3e-7.  The unit cuts off where it adds: operands
// that are both of one sign, which a layer's are not, are 7.5e-8 to 8.5e-8 too small on average, 8.7e-8 | 2.2e-7, 9.2e-8 | 9.1e-8, 9.3e-8 | 8.7e-8
// off in all (uniform), 9.6e-8 | 1.7e-7, 1.0e-7 | 7.5e-8, 1.0e-7 | 8.4e-8 (squared ReLU).
//
// The order of the sums depends on N and K alone: runs of 64 products in ascending k within a part of K, the parts' sums in ascending order
// (`parts_of`).  A row's result is the same bits whatever else is in the batch, one row or thousands.  What the batch decides is who does the
// work (`choose`): a pair takes a tile's parts one after the other, its total in the workspace in between; each part is a unit and a second
// kernel adds them up; or, with few tokens, any pieces of K are units and hand on their runs' sums, which the second kernel adds up.
// That costs many tokens some time: microseconds with the cut by M as well | now: 700 x 6144 x 2048 91 | 108, x 2048 x 8192 119 | 138, 350 x 8192 x 2048 93 | 100,
// 2,048 x 6144 x 2048 258 | 324, 700 x 8192 x 2048 174 | 170, 700 x 14336 x 2048 263 | 262; 16 x 6144 x 2048 23.3 | 24.2.
//
// A part's sum whose operands the terms may not have held (`held`: numbers that are not finite, and very small ones) is computed again with
// multiply-adds, so that it becomes what a plain product gives.
#include "linear_finish.cuh"
#include "per_device.h"
#include "sm100.cuh"
#include "terms.cuh"

#include <algorithm>

using namespace sm100;

namespace {

constexpr int BK = 64, UMMA_K = 16;
constexpr int FEATURES = 256;                           // of a pair's tile
constexpr int WARPS = 16, THREADS = 32 * WARPS;

template <int NT> struct Tile {
    static constexpr int TOKENS = NT / 2;               // of a CTA
    static constexpr int TERM_W = 128 * 128, TERM_X = TOKENS * 128;     // bytes of one term's tile
    static constexpr int STAGE = 3 * (TERM_W + TERM_X);
    static constexpr int STAGES = NT == 256 ? 2 : NT == 32 ? 4 : 3;
    static constexpr int SMEM = STAGES * STAGE + 1024 + 256;
    static constexpr int ACC = NT / 4;                  // sums of a thread
    static constexpr uint32_t TMEM = 2 * NT;
};

struct Product {
    float* C; const float *A, *W;
    const void* bias; int bias_dtype, act;
    const float *res1, *res2;
    int M, N, K;
    size_t lda, ldc, ldr;
    int m_tiles, n_tiles, parts, cut;                   // cut: units of a tile that run side by side; 1: a pair takes its parts in order
    float* partial;                                     // cut: [parts][M][N], or the runs [k-blocks][M][N]; else a tile per pair
    int32_t* status;
};

__device__ __forceinline__ bool wait_for(uint64_t* bar, uint32_t parity, volatile uint32_t* aborted, const int32_t* status) {
    for (uint32_t i = 0; i < kSpinLimit; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && (*aborted || *reinterpret_cast<const volatile int32_t*>(status) != 0)) return false;
    }
    return false;
}

// Four neighbouring numbers of a row (16-byte aligned), zeros where there are none.
__device__ __forceinline__ void fetch4(f32x2 (&r)[2], const float* p, bool have) {
    if (have) asm volatile("ld.global.v2.b64 {%0, %1}, [%2];" : "=l"(r[0]), "=l"(r[1]) : "l"(p));
    else r[0] = r[1] = 0ull;
}

// The three terms of four numbers, 8 bytes each, at dst, dst + term and dst + 2 term; of a number that has none the last is NaN.
__device__ __forceinline__ void split4(const f32x2 (&r)[2], uint32_t dst, uint32_t term) {
    uint32_t h[2], m[2], l[2];
#pragma unroll
    for (int j = 0; j < 2; ++j) terms_of(r[j], h[j], m[j], l[j]);
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst), "r"(h[0]), "r"(h[1]) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + term), "r"(m[0]), "r"(m[1]) : "memory");
    asm volatile("st.shared.v2.b32 [%0], {%1, %2};" ::"r"(dst + 2 * term), "r"(l[0]), "r"(l[1]) : "memory");
}

__device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ void tmem_load_32x8(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

// A part's sum that the terms did not hold, by multiply-adds in runs of 256 products.
__device__ __noinline__ float plain_sum(const float* __restrict__ a, const float* __restrict__ w, int k0, int k1) {
    float total = 0.f;
    while (k0 < k1) {
        float run = 0.f;
        const int end = min(k1, k0 + 256);
        for (; k0 < end; ++k0) run = fmaf(a[k0], w[k0], run);
        total += run;
    }
    return total;
}

// An arrival on a barrier of the pair's first CTA.  What it announces is read by the tensor cores, behind the fences of its proxy: no
// release over the cluster, which would wait for the loads under way.
__device__ __forceinline__ void arrive_at(uint32_t cluster_addr) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}

__device__ __forceinline__ int first_block(int kbs, int n, int i) { return (int)((long long)i * kbs / n); }

// A pair's i-th unit: the parts of its own tiles in order, or every so many of all tiles' pieces.
struct Unit { int tile, piece, f0, t0, kb0, kb1; };
__device__ __forceinline__ Unit unit_of(const Product& p, int i, int nt) {
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, kbs = (p.K + BK - 1) / BK, u = pair + i * pairs, pieces = p.cut > 1 ? p.cut : p.parts;
    const int tile = p.cut > 1 ? u / pieces : pair + i / pieces * pairs, piece = p.cut > 1 ? u % pieces : i % pieces;
    return {tile, piece, tile / p.m_tiles * FEATURES, tile % p.m_tiles * nt, first_block(kbs, pieces, piece), first_block(kbs, pieces, piece + 1)};
}

// RUNS: the runs' sums go to memory one by one, where K is cut elsewhere than between its parts (few tokens).
template <int NT, bool RUNS>
__global__ void __launch_bounds__(THREADS, 1)
linear_split_kernel(const Product p) {
    using T = Tile<NT>;
    constexpr int ACC = T::ACC, PIECE = ACC < 16 ? ACC : 16;
    constexpr uint32_t IDESC = idesc_bf16_f32(FEATURES, NT);
    extern __shared__ uint8_t smem_raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    uint64_t* full = reinterpret_cast<uint64_t*>(smem + T::STAGES * T::STAGE);     // the first CTA's: both CTAs' worker warps
    uint64_t* empty = full + T::STAGES;
    uint64_t* acc_full = empty + T::STAGES;             // [2]
    uint64_t* acc_empty = acc_full + 2;                 // [2], the first CTA's
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(acc_empty + 2);
    volatile uint32_t* aborted = tmem_slot + 1;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_ctarank();

    if (threadIdx.x == 0) {
        for (int s = 0; s < T::STAGES; ++s) { mbar_init(&full[s], 2 * WARPS); mbar_init(&empty[s], 1); }
        for (int b = 0; b < 2; ++b) { mbar_init(&acc_full[b], 1); mbar_init(&acc_empty[b], 2 * WARPS); }
        *aborted = 0;
        mbar_fence_init();
    }
    if (warp == 0) { tmem_alloc_pair(tmem_slot, T::TMEM); tmem_relinquish_pair(); }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    grid_dep_launch();

    {
        const int quad = warp & 3, group = warp >> 2;
        // A warp's share of a stage: eight rows of W, XR requests of A.  A request is four rows by 32 numbers, whole lines of memory: eight lanes
        // to a row, rows 0, 4, 1, 5 (or two more) of a group of eight, so that sixteen lanes' stores of 8 bytes meet all banks.
        constexpr int XR = NT >= 64 ? NT / 64 : 1;
        const int sub = (lane >> 4) + (lane >> 3 & 1) * 4, c4 = (lane & 7) * 4;
        // numbers 32 half + c4 of row r of a term's tile; the other half is at ^ 64, two rows on (from sub) at (^ 32) + 256
        auto place = [&](int r, int half) { return (uint32_t)(r * 128 + (((half * 4 + (c4 >> 3)) ^ (r & 7)) << 4) + (lane & 1) * 8); };
        const int x_id = warp * XR, x_first = (x_id >> 2) * 8 + (x_id >> 1 & 1) * 2 + sub;
        const uint32_t w_at = place(warp * 8 + sub, 0), x_at = 3 * T::TERM_W + place(x_first, x_id & 1);
        auto on = [&](uint32_t at, int i) { return i == 0 ? at : i == 1 ? at ^ 64u : i == 2 ? (at ^ 32u) + 256u : (at ^ 96u) + 256u; };
        const bool has_x = NT >= 64 || warp < 8;
        uint32_t full0[T::STAGES];
#pragma unroll
        for (int s = 0; s < T::STAGES; ++s) full0[s] = map_to_cta(&full[s], 0);
        const uint32_t empty0 = map_to_cta(&acc_empty[0], 0);
        const uint32_t tmem_own = tmem_base + ((uint32_t)(quad * 32) << 16) + group * ACC;
        grid_dep_wait();
        uint32_t it = 0;
        bool gave_up = false;                           // a wait ran out: no more work, but every barrier is still met
        for (int i = 0;; ++i) {
            const Unit at = unit_of(p, i, NT);
            if (at.tile >= p.m_tiles * p.n_tiles) break;
            const int f_row = at.f0 + rank * 128 + warp * 8 + sub, t_row = at.t0 + rank * T::TOKENS + x_first;
            const float* pw = p.W + (size_t)f_row * p.K + at.kb0 * BK + c4;
            const float* px = p.A + (size_t)t_row * p.lda + at.kb0 * BK + (x_id & 1) * 32 + c4;
            const bool w0 = f_row < p.N, w2 = f_row + 2 < p.N, x0 = has_x && t_row < p.M, x2 = has_x && t_row + 2 < p.M;
            f32x2 rw[4][2], rx[XR][2];
            f32x2 sum[ACC / 2];
#pragma unroll
            for (int j = 0; j < ACC / 2; ++j) sum[j] = 0ull;
            auto multiply = [&]() {                     // k-block `it`, by one thread of the pair
                const int s = it % T::STAGES, buf = it & 1;
                if (!wait_for(&acc_empty[buf], ((it >> 1) & 1) ^ 1, aborted, p.status) ||
                    !wait_for(&full[s], (it / T::STAGES) & 1, aborted, p.status)) { atomicExch(p.status, 161); *aborted = 1; return; }
                tc_fence_after_sync();
                const uint32_t w = smem_u32(smem + s * T::STAGE), x = w + 3 * T::TERM_W;
                constexpr int WT[6] = {2, 0, 1, 1, 0, 0}, XT[6] = {0, 2, 1, 0, 1, 0};      // small products first
#pragma unroll
                for (int q = 0; q < 6; ++q) {
                    const uint64_t dw = smem_desc_sw128(w + WT[q] * T::TERM_W), dx = smem_desc_sw128(x + XT[q] * T::TERM_X);
#pragma unroll
                    for (int k = 0; k < BK / UMMA_K; ++k) mma_bf16_pair(tmem_base + buf * NT, dw + 2 * k, dx + 2 * k, IDESC, q + k != 0);
                }
                mma_commit_pair(&empty[s], 3);
                mma_commit_pair(&acc_full[buf], 3);
            };
            auto take_run = [&](uint32_t run, int kb) {         // a run's sums from TMEM onto the thread's own
                const int buf = run & 1;
                if (!__all_sync(0xffffffffu, wait_for(&acc_full[buf], (run >> 1) & 1, aborted, p.status))) {
                    atomicExch(p.status, 162);
                    *aborted = 1;
                    gave_up = true;
                    return;
                }
                tc_fence_after_sync();
#pragma unroll
                for (int c = 0; c < ACC; c += PIECE) {
                    uint32_t raw[PIECE];
                    if constexpr (PIECE == 16) tmem_load_32x16(tmem_own + buf * NT + c, raw);
                    else tmem_load_32x8(tmem_own + buf * NT + c, raw);
                    tmem_load_wait();
                    if constexpr (RUNS) {
                        const int f = at.f0 + rank * 128 + quad * 32 + lane, t = at.t0 + group * ACC + c;
                        float* const to = p.partial + ((size_t)kb * p.M + t) * p.N + f;
                        if (f < p.N)
#pragma unroll
                            for (int j = 0; j < PIECE; ++j) if (t + j < p.M) to[(size_t)j * p.N] = __uint_as_float(raw[j]);
                    } else
#pragma unroll
                    for (int j = 0; j < PIECE; j += 2) sum[(c + j) / 2] = add2(sum[(c + j) / 2], pack2(__uint_as_float(raw[j]), __uint_as_float(raw[j + 1])));
                }
                tc_fence_before_sync();
                __syncwarp();
                if (lane == 0) arrive_at(empty0 + buf * 8);
            };
            int left = p.K - at.kb0 * BK - c4;          // numbers of the rows from this lane's on
            auto fetch_w = [&](int i) { fetch4(rw[i], pw + (i & 2 ? 2 * (size_t)p.K : 0) + (i & 1) * 32, (i & 2 ? w2 : w0) && left > (i & 1) * 32); };
            auto fetch_x = [&](int i) { fetch4(rx[i], px + (i & 2 ? 2 * p.lda : 0) + (i & 1) * 32, (i & 2 ? x2 : x0) && left > ((i | x_id) & 1) * 32); };
#pragma unroll
            for (int i = 0; i < 4; ++i) fetch_w(i);
#pragma unroll
            for (int i = 0; i < XR; ++i) fetch_x(i);
            for (int kb = at.kb0; kb < at.kb1 && !gave_up; ++kb, ++it) {
                const int s = it % T::STAGES;
                if (!__all_sync(0xffffffffu, wait_for(&empty[s], ((it / T::STAGES) & 1) ^ 1, aborted, p.status))) {
                    atomicExch(p.status, 163);
                    *aborted = 1;
                    gave_up = true;
                    break;
                }
                const uint32_t stage = smem_u32(smem + s * T::STAGE);
                if constexpr (NT <= 64) {               // W's lines of the k-block after the next two on their way to L2: 16 lanes, a line each
                    const int r = at.f0 + rank * 128 + warp * 8 + (lane >> 1), c = (kb + 3) * BK + (lane & 1) * 32;
                    if (lane < 16 && kb + 3 < at.kb1 && r < p.N && c < p.K) asm volatile("prefetch.global.L2 [%0];" ::"l"(p.W + (size_t)r * p.K + c));
                }
                left = kb + 1 < at.kb1 ? left - BK : 0;
                pw += BK; px += BK;
#pragma unroll
                for (int i = 0; i < 4; ++i) {           // the next k-block's numbers set out as soon as their registers are free
                    split4(rw[i], stage + on(w_at, i), T::TERM_W);
                    fetch_w(i);
                }
                if (has_x)
#pragma unroll
                    for (int i = 0; i < XR; ++i) {
                        split4(rx[i], stage + on(x_at, i), T::TERM_X);
                        fetch_x(i);
                    }
                fence_proxy_async_smem();
                __syncwarp();
                if (lane == 0) arrive_at(full0[s]);
                if (warp == 0 && rank == 0) {
                    if (elect_one()) multiply();
                    __syncwarp();
                }
                if (kb > at.kb0) take_run(it - 1, kb - 1);
            }
            if (!gave_up) take_run(it - 1, at.kb1 - 1);
            if constexpr (RUNS) continue;
            // every MMA of the unit is done: its stages hold the sums for a moment, so that the loop over them need not be unrolled
            float4* const rest = reinterpret_cast<float4*>(smem) + threadIdx.x;           // four neighbouring tokens each
            asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
            unsigned long long odd = 0ull;              // sums that the terms did not hold
#pragma unroll
            for (int j = 0; j < ACC / 4; ++j) {
                const float2 a = unpack2(sum[2 * j]), b = unpack2(sum[2 * j + 1]);
                rest[j * THREADS] = make_float4(a.x, a.y, b.x, b.y);
                odd |= (unsigned long long)(!held(a.x) | !held(a.y) << 1 | !held(b.x) << 2 | !held(b.y) << 3) << 4 * j;
            }
            asm volatile("" ::: "memory");
            const int f = at.f0 + rank * 128 + quad * 32 + lane, t = at.t0 + group * ACC, n = min(ACC, p.M - t);
            const int part = at.piece, k0 = at.kb0 * BK, k1 = min(p.K, at.kb1 * BK);
            if (f < p.N && !gave_up) {
                auto one = [&](int j) -> float& { return reinterpret_cast<float*>(rest + (j >> 2) * THREADS)[j & 3]; };
                for (; odd; odd &= odd - 1) {
                    const int j = __ffsll(odd) - 1;
                    if (j < n) one(j) = plain_sum(p.A + (size_t)(t + j) * p.lda, p.W + (size_t)f * p.K, k0, k1);
                }
                float4* const total = reinterpret_cast<float4*>(p.partial) + (size_t)blockIdx.x * (ACC / 4) * THREADS + threadIdx.x;
                if (p.cut == 1 && part > 0) {         // the pair's total so far
                    float4 before[ACC / 4];
#pragma unroll
                    for (int j = 0; j < ACC / 4; ++j) before[j] = total[j * THREADS];
#pragma unroll
                    for (int j = 0; j < ACC / 4; ++j) {
                        const float4 v = rest[j * THREADS];
                        rest[j * THREADS] = make_float4(before[j].x + v.x, before[j].y + v.y, before[j].z + v.z, before[j].w + v.w);
                    }
                }
                if (p.cut > 1) {
                    float* const to = p.partial + ((size_t)part * p.M + t) * p.N + f;
#pragma unroll 2
                    for (int j = 0; j < n; j += 4) {
                        const float4 v = rest[j / 4 * THREADS];
                        to[(size_t)j * p.N] = v.x;
                        if (j + 1 < n) to[(size_t)(j + 1) * p.N] = v.y;
                        if (j + 2 < n) to[(size_t)(j + 2) * p.N] = v.z;
                        if (j + 3 < n) to[(size_t)(j + 3) * p.N] = v.w;
                    }
                } else if (part + 1 < p.parts) {
#pragma unroll
                    for (int j = 0; j < ACC / 4; ++j) total[j * THREADS] = rest[j * THREADS];
                } else {
                    const float b = p.bias ? load_as_f32(p.bias, p.bias_dtype, f) : 0.f;
#pragma unroll 1
                    for (int j0 = 0; j0 < n; j0 += 4) {
                        const float4 four = rest[j0 / 4 * THREADS];
                        const float sums[4] = {four.x, four.y, four.z, four.w};
#pragma unroll
                        for (int j = 0; j < 4; ++j) {
                            if (j0 + j >= n) break;
                            const int row = t + j0 + j;
                            const size_t r = (size_t)row * p.ldr + f;
                            float v = sums[j];
                            if (p.bias) v += b;
                            v = apply_activation(v, p.act);
                            if (p.res1) v += p.res1[r];
                            if (p.res2) v += p.res2[r];
                            p.C[(size_t)row * p.ldc + f] = v;
                        }
                    }
                }
            }
            asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
        }
    }
    tc_fence_before_sync();
    __syncthreads();
    cluster_sync();
    if (warp == 0) tmem_dealloc_pair(tmem_base, T::TMEM);
}

// C = act(the parts' sums, in order, + bias) + residuals from the runs' sums.
constexpr int AHEAD = 32;                               // loads under way: one thread walks all of K
__global__ void __launch_bounds__(128)
split_join_runs_kernel(const Product p) {
    const size_t mn = (size_t)p.M * p.N;
    const int kbs = (p.K + BK - 1) / BK;
    grid_dep_launch();
    grid_dep_wait();
    for (size_t e = (size_t)blockIdx.x * blockDim.x + threadIdx.x; e < mn; e += (size_t)gridDim.x * blockDim.x) {
        const int row = (int)(e / p.N), f = (int)(e % p.N);
        float total = 0.f, sum = 0.f;
        int part = 0, k0 = 0, k1 = first_block(kbs, p.parts, 1);
        for (int base = 0; base < kbs; base += AHEAD) {
            float v[AHEAD];
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) v[i] = base + i < kbs ? p.partial[(size_t)(base + i) * mn + e] : 0.f;
#pragma unroll
            for (int i = 0; i < AHEAD; ++i) {
                if (base + i >= kbs) break;
                sum += v[i];
                if (base + i + 1 == k1) {               // a part's end
                    if (!held(sum)) sum = plain_sum(p.A + (size_t)row * p.lda, p.W + (size_t)f * p.K, k0 * BK, min(p.K, k1 * BK));
                    total += sum;
                    sum = 0.f;
                    k0 = k1;
                    k1 = first_block(kbs, p.parts, ++part + 1);
                }
            }
        }
        finish(p.C, total, row, f, p.bias, p.bias_dtype, p.act, p.res1, p.res2, p.ldc, p.ldr);
    }
}

// Pairs of these blocks that the current device runs at once.  The kernel's limit of shared memory, set on the way, is the device's own too.
template <int NT, bool RUNS>
int max_pairs(int* pairs) {
    static PerDevice known;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e == cudaSuccess) *pairs = known.get(dev, [&] {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(2); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Tile<NT>::SMEM;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr; cfg.numAttrs = 1;
        int n = 0;
        e = cudaFuncSetAttribute(linear_split_kernel<NT, RUNS>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<NT>::SMEM);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, linear_split_kernel<NT, RUNS>, &cfg);
        return e == cudaSuccess ? n : 0;
    });
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_split: %s", cudaGetErrorString(e));
    return *pairs > 0 ? QS_OK : qs_fail(QS_ERR_INTERNAL, "linear_split: this device runs no pair of these blocks");
}

constexpr int PAIRS = 74;                               // of a B200

template <int NT, bool RUNS>
int launch(const Product& p, cudaStream_t stream) {
    int pairs = 0;
    const int rc = max_pairs<NT, RUNS>(&pairs);
    if (rc != QS_OK) return rc;
    const long long units = (long long)p.m_tiles * p.n_tiles * p.cut;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)std::min<long long>(units, std::min(pairs, PAIRS))); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Tile<NT>::SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, linear_split_kernel<NT, RUNS>, p);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_split: %s", cudaGetErrorString(e));
    return qs_check_launch("linear_split");
}

// The parts of K, whose sums are added in order: by N and K alone, so that a row's result is the same bits whatever else is in the batch.  As many as
// put a unit on every pair where there is one tile of tokens, of ten k-blocks at least.
int parts_of(int N, int K) {
    const int n_tiles = (N + FEATURES - 1) / FEATURES, kbs = (K + BK - 1) / BK;
    return std::max(1, std::min(kbs / 10, PAIRS / n_tiles));
}

// Tokens of a tile and who works on its parts: one pair in order (cut = 1), a unit per part, joined by a kernel behind, or, with few tokens, any
// pieces, whose runs are joined one by one.  The least microseconds: rounds of units over the pairs, a unit's k-blocks and its two ends (all
// measured), what the sums' way through memory costs.
struct Form { int nt, parts, cut; bool runs; };
Form choose(int M, int N, int K) {
    constexpr int NTS[4] = {32, 64, 128, 256};
    constexpr double BLOCK[4] = {1.3, 1.33, 1.6, 2.48}, ENDS[4] = {2.5, 3.0, 5.0, 9.0}, RUN_ENDS = 1.5, JOIN = 3.0, JOIN_RUNS = 4.0, BYTES = 6e6;
    const int kbs = (K + BK - 1) / BK, parts = parts_of(N, K), per = (kbs + parts - 1) / parts;
    const long long mn = (long long)M * N;
    Form best = {256, parts, 1, false};
    double least = 1e30;
    for (int i = 0; i < 4; ++i) {
        const long long tiles = (long long)((M + NTS[i] - 1) / NTS[i]) * ((N + FEATURES - 1) / FEATURES);
        auto rounds = [&](int cut) { return (double)((tiles * cut + PAIRS - 1) / PAIRS); };
        const double alone = rounds(1) * (kbs * BLOCK[i] + parts * ENDS[i]);
        if (alone < least) { least = alone; best = {NTS[i], parts, 1, false}; }
        if (parts > 1 && mn * parts <= (1ll << 26)) {
            const double side = rounds(parts) * (per * BLOCK[i] + ENDS[i]) + JOIN + mn * parts * 4 / BYTES;
            if (side < least) { least = side; best = {NTS[i], parts, parts, false}; }
        }
        if (NTS[i] > 64 || mn * kbs > (1ll << 24)) continue;
        for (int cut = 2; cut <= kbs && tiles * cut <= 4 * PAIRS; ++cut) {
            const double runs = rounds(cut) * ((kbs + cut - 1) / cut * BLOCK[i] + RUN_ENDS) + JOIN_RUNS + mn * kbs * 8 / BYTES;
            if (runs < least) { least = runs; best = {NTS[i], parts, cut, true}; }
        }
    }
    return best;
}
long long scratch_of(const Form& f, int M, int N, int K) {
    const long long mn = (long long)M * N;
    if (f.cut > 1) return mn * (f.runs ? (K + BK - 1) / BK : f.parts);
    return f.parts > 1 ? (long long)PAIRS * FEATURES * f.nt : 0;
}

}  // namespace

// How many floats of workspace `qs_linear_split` takes for this product (0: none).
QS_API long long qs_linear_split_scratch(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    return scratch_of(choose(M, N, K), M, N, K);
}

// How a product is worked on: tokens of a tile, parts of K, units of a tile side by side, whether these hand on runs.
QS_API int qs_linear_split_form(int M, int N, int K, int* form) {
    QS_REQUIRE(M > 0 && N > 0 && K > 0 && form, "linear_split: bad sizes M=%d N=%d K=%d", M, N, K);
    const Form f = choose(M, N, K);
    form[0] = f.nt; form[1] = f.parts; form[2] = f.cut; form[3] = f.runs;
    return QS_OK;
}

// All operands float32.  A and W 16-byte aligned, K and lda multiples of four.  ws: `qs_linear_split_scratch` floats.
// status: device int32 that receives a non-zero code if a bounded wait inside the kernel ran out.
QS_API int qs_linear_split(float* C, const float* A, const float* W, const void* bias, int bias_dtype, int act, const float* res1, const float* res2,
                           int M, int N, int K, long long lda, long long ldc, long long ldr, float* ws, long long ws_floats, int32_t* status,
                           cudaStream_t stream) {
    if (M == 0 || N == 0) return QS_OK;
    QS_REQUIRE(M > 0 && N > 0 && K > 0, "linear_split: bad sizes M=%d N=%d K=%d", M, N, K);
    QS_REQUIRE(K % 4 == 0 && lda % 4 == 0 && lda >= K && ldc >= N, "linear_split: K=%d and the row stride %lld must be multiples of four", K, lda);
    QS_REQUIRE(((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0, "linear_split: operands must be 16-byte aligned");
    const Form f = choose(M, N, K);
    const long long floats = scratch_of(f, M, N, K);
    QS_REQUIRE(floats == 0 || (ws && ws_floats >= floats), "linear_split: %lld floats of workspace instead of %lld", ws_floats, floats);
    Product p = {};
    p.C = C; p.A = A; p.W = W; p.bias = bias; p.bias_dtype = bias_dtype; p.act = act; p.res1 = res1; p.res2 = res2; p.M = M; p.N = N; p.K = K;
    p.lda = (size_t)lda; p.ldc = (size_t)ldc; p.ldr = (size_t)ldr; p.status = status;
    p.parts = f.parts; p.cut = f.cut;
    p.m_tiles = (M + f.nt - 1) / f.nt; p.n_tiles = (N + FEATURES - 1) / FEATURES;
    QS_REQUIRE((long long)p.m_tiles * p.n_tiles * std::max(p.parts, p.cut) <= 0x3fffffffll, "linear_split: %d x %d outputs", M, N);
    p.partial = floats ? ws : nullptr;
    const int rc = f.runs ? (f.nt == 32 ? launch<32, true>(p, stream) : launch<64, true>(p, stream))
                 : f.nt == 32 ? launch<32, false>(p, stream) : f.nt == 64 ? launch<64, false>(p, stream)
                 : f.nt == 128 ? launch<128, false>(p, stream) : launch<256, false>(p, stream);
    if (rc != QS_OK || f.cut == 1) return rc;
    const size_t mn = (size_t)M * N;
    if (f.runs) {
        const cudaError_t e = qs_launch_dependent(split_join_runs_kernel, dim3((unsigned)std::min<size_t>(mn / 128 + 1, 16 * 148)), dim3(128), 0, stream, p);
        if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_split: %s", cudaGetErrorString(e));
    } else {
        linear_join_kernel<float, float><<<(unsigned)std::min<size_t>(mn / 256 + 1, 8 * 148), 256, 0, stream>>>(C, ws, f.parts, bias, bias_dtype, act, res1, res2, M, N,
                                                                                                                (size_t)ldc, (size_t)ldr);
    }
    return qs_check_launch("linear_split");
}
