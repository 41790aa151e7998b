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
// k-block: fetch, split, barrier of the pair, MMAs, sums (700 x 6144 x 2048: 96 us, 412 there; leaving out the loads gives 84, the sums'
// way to registers 84, all but barriers, stores and MMAs 82).  Loads four rows of whole 128-byte lines at a time: eight rows of 32 bytes
// per lane took 40 wavefronts instead of 4 each; loads set out as soon as their registers are free: 96 against 102 us
// with all of them behind the barrier; two k-blocks under way for few tokens: no gain, more registers.  Few rows (up to 64 or so) are bound by the latency of that
// chain: 64 x 6144 x 2048 36 us (60).
//
// Error against float64, 2-norm, normal numbers, this | CUDA cores: K = 256 8.8e-8 | 2.9e-7, 2,048 1.1e-7 | 2.9e-7, 8,192 1.5e-7 |
// 3.1e-7.
//
// Few tiles: K is cut, the parts' sums go to `partial` and a second kernel adds them in order.
//
// Numbers that are not finite (or round to infinity as bfloat16) have no such terms: their last one is NaN, and with it every sum they
// take part in.  Such a sum is computed again with multiply-adds, so that it becomes what a plain product gives.
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
    int m_tiles, n_tiles, splits;
    float* partial;                                     // [splits][M][N], or null
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

// A sum that the terms gave no number for, by multiply-adds in runs of 256 products.
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

struct Unit { int f0, t0, kb0, kb1, part; };
__device__ __forceinline__ Unit unit_of(const Product& p, int u, int nt) {
    const int part = u % p.splits, tile = u / p.splits, kbs = (p.K + BK - 1) / BK;
    return {tile / p.m_tiles * FEATURES, tile % p.m_tiles * nt, (int)((long long)part * kbs / p.splits), (int)((long long)(part + 1) * kbs / p.splits), part};
}

template <int NT>
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
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, units = p.m_tiles * p.n_tiles * p.splits;

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
        for (int u = pair; u < units; u += pairs) {
            const Unit at = unit_of(p, u, NT);
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
            auto take_run = [&](uint32_t run) {         // a run's sums from TMEM onto the thread's own
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
                if (kb > at.kb0) take_run(it - 1);
            }
            if (!gave_up) take_run(it - 1);
            // every MMA of the unit is done: its stages hold the sums for a moment, so that the loop over them need not be unrolled
            float* rest = reinterpret_cast<float*>(smem) + threadIdx.x;
            asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory");
#pragma unroll
            for (int j = 0; j < ACC; j += 2) {
                const float2 v = unpack2(sum[j / 2]);
                rest[j * THREADS] = v.x;
                rest[(j + 1) * THREADS] = v.y;
            }
            const int f = at.f0 + rank * 128 + quad * 32 + lane, t = at.t0 + group * ACC, n = min(ACC, p.M - t);
            if (f < p.N && !gave_up) {
                const float b = p.bias ? load_as_f32(p.bias, p.bias_dtype, f) : 0.f;
#pragma unroll 4
                for (int j = 0; j < n; ++j) {
                    float v = rest[j * THREADS];
                    if (!(fabsf(v) <= 3.402823466e38f)) v = plain_sum(p.A + (size_t)(t + j) * p.lda, p.W + (size_t)f * p.K, at.kb0 * BK, min(p.K, at.kb1 * BK));
                    if (p.partial) { p.partial[((size_t)at.part * p.M + t + j) * p.N + f] = v; continue; }
                    const size_t r = (size_t)(t + j) * p.ldr + f;
                    if (p.bias) v += b;
                    v = apply_activation(v, p.act);
                    if (p.res1) v += p.res1[r];
                    if (p.res2) v += p.res2[r];
                    p.C[(size_t)(t + j) * p.ldc + f] = v;
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

// Pairs of these blocks that the current device runs at once.  The kernel's limit of shared memory, set on the way, is the device's own too.
template <int NT>
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
        e = cudaFuncSetAttribute(linear_split_kernel<NT>, cudaFuncAttributeMaxDynamicSharedMemorySize, Tile<NT>::SMEM);
        if (e == cudaSuccess) e = cudaOccupancyMaxActiveClusters(&n, linear_split_kernel<NT>, &cfg);
        return e == cudaSuccess ? n : 0;
    });
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_split: %s", cudaGetErrorString(e));
    return *pairs > 0 ? QS_OK : qs_fail(QS_ERR_INTERNAL, "linear_split: this device runs no pair of these blocks");
}

template <int NT>
int launch(Product p, cudaStream_t stream) {
    int pairs = 0;
    const int rc = max_pairs<NT>(&pairs);
    if (rc != QS_OK) return rc;
    const long long units = (long long)p.m_tiles * p.n_tiles * p.splits;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)std::min<long long>(units, pairs)); cfg.blockDim = dim3(THREADS); cfg.dynamicSmemBytes = Tile<NT>::SMEM; cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2; attr[0].val.clusterDim.y = 1; attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr; cfg.numAttrs = 2;
    const cudaError_t e = cudaLaunchKernelEx(&cfg, linear_split_kernel<NT>, p);
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_split: %s", cudaGetErrorString(e));
    return qs_check_launch("linear_split");
}

// Tokens of a tile and parts of K: the least of rounds of units over the 74 pairs, a unit's share of K times the cycles of a
// k-block (measured), and what the sums of a cut cost.
struct Form { int nt, splits; };
Form choose(int M, int N, int K, bool may_split) {
    constexpr int PAIRS = 74, NTS[4] = {32, 64, 128, 256};
    constexpr double CYCLES[4] = {2400.0, 2500.0, 3000.0, 4700.0};
    Form best = {256, 1};
    double best_cost = 1e30;
    const int kbs = (K + BK - 1) / BK;
    for (int i = 0; i < 4; ++i) {
        const long long tiles = (long long)((M + NTS[i] - 1) / NTS[i]) * ((N + FEATURES - 1) / FEATURES);
        for (int splits = 1; splits <= kbs && splits <= PAIRS; ++splits) {
            if (splits > 1 && (!may_split || tiles * splits > 4 * PAIRS || (long long)M * N * splits > (1ll << 26))) break;
            const long long rounds = (tiles * splits + PAIRS - 1) / PAIRS;
            double cost = rounds * (((kbs + splits - 1) / splits) * CYCLES[i] + 4000.0);
            if (splits > 1) cost += 4000.0 + (double)M * N * splits / 1000.0;
            if (cost < best_cost) { best_cost = cost; best = {NTS[i], splits}; }
        }
    }
    return best;
}

}  // namespace

// How many floats of workspace `qs_linear_split` uses for this product (0: none).
QS_API long long qs_linear_split_scratch(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    const Form f = choose(M, N, K, true);
    return f.splits > 1 ? (long long)f.splits * M * N : 0;
}

// All operands float32.  A and W 16-byte aligned, K and lda multiples of four.  ws: `qs_linear_split_scratch` floats; with fewer (or none) K is
// not cut.  status: device int32 that receives a non-zero code if a bounded wait inside the kernel ran out.
QS_API int qs_linear_split(float* C, const float* A, const float* W, const void* bias, int bias_dtype, int act, const float* res1, const float* res2,
                           int M, int N, int K, long long lda, long long ldc, long long ldr, float* ws, long long ws_floats, int32_t* status,
                           cudaStream_t stream) {
    if (M == 0 || N == 0) return QS_OK;
    QS_REQUIRE(M > 0 && N > 0 && K > 0, "linear_split: bad sizes M=%d N=%d K=%d", M, N, K);
    QS_REQUIRE(K % 4 == 0 && lda % 4 == 0 && lda >= K && ldc >= N, "linear_split: K=%d and the row stride %lld must be multiples of four", K, lda);
    QS_REQUIRE(((uintptr_t)A % 16) == 0 && ((uintptr_t)W % 16) == 0, "linear_split: operands must be 16-byte aligned");
    Form f = choose(M, N, K, true);
    if (f.splits > 1 && (!ws || ws_floats < (long long)f.splits * M * N)) f = choose(M, N, K, false);
    Product p = {};
    p.C = C; p.A = A; p.W = W; p.bias = bias; p.bias_dtype = bias_dtype; p.act = act; p.res1 = res1; p.res2 = res2; p.M = M; p.N = N; p.K = K;
    p.lda = (size_t)lda; p.ldc = (size_t)ldc; p.ldr = (size_t)ldr; p.status = status; p.splits = f.splits;
    p.m_tiles = (M + f.nt - 1) / f.nt; p.n_tiles = (N + FEATURES - 1) / FEATURES;
    QS_REQUIRE((long long)p.m_tiles * p.n_tiles * p.splits <= 0x7fffffffll, "linear_split: %d x %d outputs", M, N);
    p.partial = f.splits > 1 ? ws : nullptr;
    const int rc = f.nt == 32 ? launch<32>(p, stream) : f.nt == 64 ? launch<64>(p, stream) : f.nt == 128 ? launch<128>(p, stream) : launch<256>(p, stream);
    if (rc != QS_OK || !p.partial) return rc;
    const size_t mn = (size_t)M * N;
    const int blocks = (int)std::min<size_t>(mn / 256 + 1, 8 * 148);
    linear_join_kernel<float, float><<<blocks, 256, 0, stream>>>(C, ws, f.splits, bias, bias_dtype, act, res1, res2, M, N, (size_t)ldc, (size_t)ldr);
    return qs_check_launch("linear_split");
}
