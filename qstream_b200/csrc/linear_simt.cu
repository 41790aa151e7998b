// C = act(A W^T + bias) + res1 + res2 on the CUDA cores, accumulating in true
// 32-bit (FFMA; no tensor-core or reduced-precision matrix mode).
//
// This is the product for what the tensor-core kernels do not take: a matrix stored
// in 32-bit used with bfloat16 activations, short sums and odd row strides of the
// float32 engine (whose other products linear_split.cu takes), its routed experts.  A: [M, K] row-major (row stride lda), W: [N, K]
// row-major, weight rows = outputs, QStream's matvec convention
// (include/qsf/kernels.h:53-58).  Each output element sums its K products in
// ascending k inside one thread, so a row's result does not depend on M or on
// which other rows are in the batch.  The sum is taken in two levels: runs of 256
// products in one accumulator, the runs' sums in a second one, so that the rounding
// error grows with sqrt(256) + sqrt(K / 256) instead of sqrt(K) (at K = 16384 a
// fifth of the single accumulator's error).
//
// The order of the sums is the same in every form below (tile sizes, cut over the runs or not), so the
// choice of the form by M, N and K never changes a bit of the result.
#include "linear_finish.cuh"

namespace {

constexpr int RUN = 256;                                   // products per first-level run

// Elements c .. c + 3 of a row as 32-bit numbers, zeros from `end` on.  `vec`: the row starts aligned and `end` is a
// multiple of four, so that a piece is whole or absent.
template <typename T>
__device__ __forceinline__ float4 load4(const T* __restrict__ row, int c, int end, bool vec) {
    if (c >= end) return make_float4(0.f, 0.f, 0.f, 0.f);
    if (vec) {
        if constexpr (sizeof(T) == 4) return *reinterpret_cast<const float4*>(row + c);
        const uint2 u = *reinterpret_cast<const uint2*>(row + c);
        return make_float4(__uint_as_float(u.x << 16), __uint_as_float(u.x & 0xffff0000u), __uint_as_float(u.y << 16), __uint_as_float(u.y & 0xffff0000u));
    }
    return make_float4(to_f32(row[c]), c + 1 < end ? to_f32(row[c + 1]) : 0.f, c + 2 < end ? to_f32(row[c + 2]) : 0.f,
                       c + 3 < end ? to_f32(row[c + 3]) : 0.f);
}

// A block computes a tile of BM x BN outputs, a thread TM x TN of them (rows in groups of four, columns in groups of four,
// so that a warp's 16-byte reads of a staged row touch neighbouring addresses).  The next k-tile's elements travel to
// registers while the present one is multiplied; shared memory holds two tiles, one barrier per tile.  The second-level
// sums rest in shared memory (touched once per 256 products).
//
// `partial` null: the block walks all of K.  Else (few tiles: blockIdx.z takes `runs_per` of the runs) every run's
// sum goes to partial[run][M][N] and `linear_join_kernel` adds them in order.
//
// Bound by multiply-add issue and the shared-memory reads beside it (four 16-byte reads per 32 paired multiply-adds): 53
// TFLOP/s of the CUDA cores' 74.5 at 2048 x 16384 x 4096 (5.2 ms; the 64 x 64 tiles of four by four per thread that stood
// here before: 12.7 ms), 43 at 700 x 6144 x 2048 (0.41 ms; 0.93).  Plain instead of paired multiply-adds: 6.2 ms; 8 x 16
// per thread: 5.3; every lane fetching from a row of its own: 6.3.
template <typename TA, typename TW, typename TC, int BM, int BN, int BK, int TM, int TN, int MIN_BLOCKS>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MIN_BLOCKS)
linear_tile_kernel(TC* __restrict__ C, const TA* __restrict__ A, const TW* __restrict__ W,
                   const void* __restrict__ bias, int bias_dtype, int act,
                   const TA* __restrict__ res1, const TA* __restrict__ res2,
                   int M, int N, int K, size_t lda, size_t ldc, size_t ldr, int vec_a, int vec_w,
                   float* __restrict__ partial, int runs_per) {
    constexpr int THREADS = (BM / TM) * (BN / TN), WARPS = THREADS / 32, RUN_TILES = RUN / BK;
    constexpr int PA = BM < 32 ? 32 : BM, PW = BN;          // a staged tile is [BK][rows], its columns swizzled (see `stage`)
    constexpr int KJ = BK / 16;
    constexpr int A_JOBS = BM / 8 * KJ, W_JOBS = BN / 8 * KJ;   // a job: 8 rows x 16 k, one warp; four lanes share a row's 16 k
    constexpr int A_PER = (A_JOBS + WARPS - 1) / WARPS, W_PER = (W_JOBS + WARPS - 1) / WARPS;
    constexpr int GM = TM / 4, GN = TN / 4;
    extern __shared__ __align__(16) float smem[];
    float* sA = smem;                                       // [2][BK][PA]
    float* sW = sA + 2 * BK * PA;                           // [2][BK][PW]
    float* sT = sW + 2 * BK * PW;                           // [TM * TN][THREADS]
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the threads of a warp form 4 x 8: 4 row groups, 8 column groups
    constexpr int COLS = BN / TN;                           // column groups of the block
    const int wx = warp % (COLS / 8), wy = warp / (COLS / 8);
    const int tx = wx * 8 + (lane & 7), ty = wy * 4 + (lane >> 3);
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int n_tiles = (K + BK - 1) / BK;
    const int first = blockIdx.z * runs_per * RUN_TILES, last = min(n_tiles, first + runs_per * RUN_TILES);

    f32x2 acc[TM][TN / 2];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN / 2; ++j) acc[i][j] = 0ull;
    const bool totals = !partial && n_tiles > RUN_TILES;
    if (totals)
#pragma unroll
        for (int e = 0; e < TM * TN; ++e) sT[e * THREADS + tid] = 0.f;

    float4 ra[A_PER], rw[W_PER];
    const int c4 = (lane & 3) * 4;                          // the lane's four k of a job
    auto fetch = [&](int tile) {
        const int k0 = tile * BK;
#pragma unroll
        for (int p = 0; p < A_PER; ++p) {
            const int job = warp + p * WARPS, gm = m0 + job / KJ * 8 + (lane >> 2);
            ra[p] = job < A_JOBS && gm < M ? load4(A + (size_t)gm * lda, k0 + job % KJ * 16 + c4, K, vec_a) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int p = 0; p < W_PER; ++p) {
            const int job = warp + p * WARPS, gn = n0 + job / KJ * 8 + (lane >> 2);
            rw[p] = job < W_JOBS && gn < N ? load4(W + (size_t)gn * K, k0 + job % KJ * 16 + c4, K, vec_w) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    // transposed; column r of row k lies at r ^ 8 (k / 4 mod 4), so that the four lanes of a row write to different banks
    auto stage = [&](int buf) {
#pragma unroll
        for (int p = 0; p < A_PER; ++p) {
            const int job = warp + p * WARPS, r = (job / KJ * 8 + (lane >> 2)) ^ (c4 * 2);
            if (job < A_JOBS) {
                float* d = sA + (buf * BK + job % KJ * 16 + c4) * PA + r;
                d[0] = ra[p].x; d[PA] = ra[p].y; d[2 * PA] = ra[p].z; d[3 * PA] = ra[p].w;
            }
        }
#pragma unroll
        for (int p = 0; p < W_PER; ++p) {
            const int job = warp + p * WARPS, r = (job / KJ * 8 + (lane >> 2)) ^ (c4 * 2);
            if (job < W_JOBS) {
                float* d = sW + (buf * BK + job % KJ * 16 + c4) * PW + r;
                d[0] = rw[p].x; d[PW] = rw[p].y; d[2 * PW] = rw[p].z; d[3 * PW] = rw[p].w;
            }
        }
    };
    constexpr int ROW_STEP = BM / GM, COL_STEP = BN / GN;   // a thread's groups of four lie this far apart
    auto row_of = [&](int i) { return (i / 4) * ROW_STEP + ty * 4 + (i & 3); };
    auto col_of = [&](int j) { return (j / 4) * COL_STEP + tx * 4 + (j & 3); };

    fetch(first);
    stage(0);
    __syncthreads();
    int in_run = 0, run = blockIdx.z * runs_per;
    for (int tile = first; tile < last; ++tile) {
        const int buf = (tile - first) & 1;
        if (tile + 1 < last) fetch(tile + 1);
#pragma unroll 16
        for (int k = 0; k < BK; ++k) {
            float a[TM];
            f32x2 w[TN / 2];
#pragma unroll
            for (int g = 0; g < GM; ++g) {
                const float4 x = *reinterpret_cast<const float4*>(sA + (buf * BK + k) * PA + ((g * ROW_STEP + ty * 4) ^ (k / 4 % 4 * 8)));
                a[4 * g] = x.x; a[4 * g + 1] = x.y; a[4 * g + 2] = x.z; a[4 * g + 3] = x.w;
            }
#pragma unroll
            for (int g = 0; g < GN; ++g) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(sW + (buf * BK + k) * PW + ((g * COL_STEP + tx * 4) ^ (k / 4 % 4 * 8)));
                w[2 * g] = x.x; w[2 * g + 1] = x.y;
            }
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const f32x2 aa = pack2(a[i], a[i]);
#pragma unroll
                for (int j = 0; j < TN / 2; ++j) acc[i][j] = fma2(aa, w[j], acc[i][j]);
            }
        }
        if (tile + 1 < last) stage(buf ^ 1);
        if (++in_run == RUN_TILES) {                         // a run is complete: on to the second level
            in_run = 0;
            if (totals) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) {
                        const float2 v = unpack2(acc[i][j]);
                        float* t = sT + (i * TN + 2 * j) * THREADS + tid;
                        t[0] += v.x;
                        t[THREADS] += v.y;
                        acc[i][j] = 0ull;
                    }
            } else if (partial) {
#pragma unroll
                for (int i = 0; i < TM; ++i)
#pragma unroll
                    for (int j = 0; j < TN / 2; ++j) {
                        const float2 v = unpack2(acc[i][j]);
                        const int gm = m0 + row_of(i), gn = n0 + col_of(2 * j);
                        float* t = partial + ((size_t)run * M + gm) * N + gn;
                        if (gm < M && gn < N) t[0] = v.x;
                        if (gm < M && gn + 1 < N) t[1] = v.y;
                        acc[i][j] = 0ull;
                    }
                ++run;
            }
        }
        __syncthreads();
    }
    if (partial && in_run == 0) return;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + row_of(i);
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + col_of(j);
            const float2 pair = unpack2(acc[i][j / 2]);
            float v = (j & 1) ? pair.y : pair.x;
            if (gm >= M || gn >= N) continue;
            if (partial) { partial[((size_t)run * M + gm) * N + gn] = v; continue; }
            if (totals) v = sT[(i * TN + j) * THREADS + tid] + v;
            finish(C, v, gm, gn, bias, bias_dtype, act, res1, res2, ldc, ldr);
        }
    }
}

constexpr int SMS = 148;

// Which tile, and into how many ranges of runs K is cut: the least of a model of the busiest SM's time.  A block of a form
// alone on its SM does FORM_ONE multiply-adds per cycle, FORM_FULL when all FORM_BLOCKS that fit are there (measured on
// grids that put one, and all, on every SM); each round of blocks costs about 2,500 cycles of filling and storing,
// and a cut the way of the runs' sums through memory and one more launch.  Measured in microseconds (M x N x K; 128 x 128,
// 64 x 64, 16 x 128 tiles, best cut | not cut): 700 x 2048 x 8192: 550, 550, - | 876, 1001, -; 150 x 2048 x 2048: 62, 55, - |
// 238, 195, -; 16 x 6144 x 2048: -, 52, 31 | -, 187, 80; 700 x 6144 x 2048: 426, 419, - | 410, 540, -.
struct Form { int tile, split; };
constexpr int N_FORMS = 3;
constexpr int FORM_BM[N_FORMS] = {128, 64, 16}, FORM_BN[N_FORMS] = {128, 64, 128}, FORM_BLOCKS[N_FORMS] = {2, 7, 4};
constexpr double FORM_ONE[N_FORMS] = {71.0, 19.0, 27.0}, FORM_FULL[N_FORMS] = {88.0, 77.0, 60.0};

Form choose(int M, int N, int K, bool may_split) {
    Form best = {0, 1};
    double best_cost = 1e30;
    const int runs = (K + RUN - 1) / RUN;
    for (int f = 0; f < N_FORMS; ++f) {
        if ((M + FORM_BM[f] - 1) / FORM_BM[f] > 65535) continue;        // the grid's limit
        const long long tiles = (long long)((M + FORM_BM[f] - 1) / FORM_BM[f]) * ((N + FORM_BN[f] - 1) / FORM_BN[f]);
        for (int split = 1; split <= runs; ++split) {
            if (split > 1 && (!may_split || tiles >= 4 * SMS || (long long)M * N * runs > (1ll << 26))) break;   // at most 256 MB of sums
            const int per = (runs + split - 1) / split;
            if ((runs + per - 1) / per != split) continue;  // the same cut as a smaller count
            const long long on_sm = (tiles * split + SMS - 1) / SMS, rounds = on_sm / FORM_BLOCKS[f], rest = on_sm % FORM_BLOCKS[f];
            const double block = (double)FORM_BM[f] * FORM_BN[f] * (split == 1 ? K : per * RUN);
            double cost = rounds * (FORM_BLOCKS[f] * block / FORM_FULL[f] + 2500.0);
            if (rest) cost += rest * block / (rest * FORM_ONE[f] < FORM_FULL[f] ? rest * FORM_ONE[f] : FORM_FULL[f]) + 2500.0;
            if (split > 1) cost += 5000.0 + (double)M * N * runs / 1000.0;
            if (cost < best_cost) { best_cost = cost; best = {f, split}; }
        }
    }
    return best;
}

template <typename TA, typename TW, typename TC>
int launch(void* C, const void* A, const void* W, const void* bias, int bias_dtype, int act,
           const void* res1, const void* res2, int M, int N, int K, long long lda, long long ldc,
           long long ldr, float* ws, long long ws_floats, cudaStream_t stream) {
    const int runs = (K + RUN - 1) / RUN;
    const Form form = choose(M, N, K, ws && ws_floats >= (long long)runs * M * N);
    const int f = form.tile, split = form.split;
    const int per = (runs + split - 1) / split;
    const int vec_a = K % 4 == 0 && lda % 4 == 0 && ((uintptr_t)A % (4 * sizeof(TA))) == 0;
    const int vec_w = K % 4 == 0 && ((uintptr_t)W % (4 * sizeof(TW))) == 0;
    float* partial = split > 1 ? ws : nullptr;
    cudaError_t e = cudaSuccess;
#define GO(BM_, BN_, BK_, TM_, TN_, MB_) do { \
        constexpr int threads = (BM_ / TM_) * (BN_ / TN_); \
        const size_t smem = (size_t)(2 * BK_ * ((BM_ < 32 ? 32 : BM_) + BN_) + (!partial && K > RUN ? TM_ * TN_ * threads : 0)) * sizeof(float); \
        auto kernel = linear_tile_kernel<TA, TW, TC, BM_, BN_, BK_, TM_, TN_, MB_>; \
        if (smem > 48 * 1024) e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); \
        if (e == cudaSuccess) kernel<<<dim3((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_, split), threads, smem, stream>>>( \
            (TC*)C, (const TA*)A, (const TW*)W, bias, bias_dtype, act, (const TA*)res1, (const TA*)res2, M, N, K, \
            (size_t)lda, (size_t)ldc, (size_t)ldr, vec_a, vec_w, partial, per); } while (0)
    if (f == 0) GO(128, 128, 16, 8, 8, 2);
    else if (f == 1) GO(64, 64, 16, 8, 8, 7);
    else GO(16, 128, 32, 4, 4, 4);
#undef GO
    if (e != cudaSuccess) return qs_fail(QS_ERR_INTERNAL, "linear_simt: %s", cudaGetErrorString(e));
    if (partial) {
        const size_t mn = (size_t)M * N;
        const int blocks = (int)(mn / 256 + 1 < 8 * SMS ? mn / 256 + 1 : 8 * SMS);
        linear_join_kernel<TA, TC><<<blocks, 256, 0, stream>>>((TC*)C, partial, runs, bias, bias_dtype, act, (const TA*)res1, (const TA*)res2,
                                                               M, N, (size_t)ldc, (size_t)ldr);
    }
    return qs_check_launch("linear_simt");
}

}  // namespace

// How many floats of workspace `qs_linear_simt` uses for this product (0: none).
QS_API long long qs_linear_simt_scratch(int M, int N, int K) {
    if (M <= 0 || N <= 0 || K <= 0) return 0;
    return choose(M, N, K, true).split > 1 ? (long long)((K + RUN - 1) / RUN) * M * N : 0;
}

// a_dtype: type of A, res1, res2.  c_dtype: type of C (a_dtype, or float32 for logits).  ws: `qs_linear_simt_scratch`
// floats; with fewer (or none) the product runs in a slower form with the same result.
QS_API int qs_linear_simt(void* C, int c_dtype, const void* A, int a_dtype, const void* W, int w_dtype,
                          const void* bias, int bias_dtype, int act, const void* res1, const void* res2,
                          int M, int N, int K, long long lda, long long ldc, long long ldr, float* ws, long long ws_floats,
                          cudaStream_t stream) {
    if (M == 0 || N == 0) return QS_OK;
    QS_REQUIRE(M > 0 && N > 0 && K > 0, "linear: bad sizes M=%d N=%d K=%d", M, N, K);
    QS_REQUIRE(lda >= K && ldc >= N, "linear: row strides lda=%lld ldc=%lld below K=%d N=%d", lda, ldc, K, N);
    QS_REQUIRE((M + 63) / 64 <= 65535, "linear: M=%d exceeds the grid", M);
#define GO(TA, TW, TC) return launch<TA, TW, TC>(C, A, W, bias, bias_dtype, act, res1, res2, M, N, K, lda, ldc, ldr, ws, ws_floats, stream)
    typedef __nv_bfloat16 bf16;
    if (a_dtype == QS_F32 && w_dtype == QS_F32 && c_dtype == QS_F32) GO(float, float, float);
    if (a_dtype == QS_F32 && w_dtype == QS_BF16 && c_dtype == QS_F32) GO(float, bf16, float);
    if (a_dtype == QS_BF16 && w_dtype == QS_BF16 && c_dtype == QS_BF16) GO(bf16, bf16, bf16);
    if (a_dtype == QS_BF16 && w_dtype == QS_BF16 && c_dtype == QS_F32) GO(bf16, bf16, float);
    if (a_dtype == QS_BF16 && w_dtype == QS_F32 && c_dtype == QS_BF16) GO(bf16, float, bf16);
    if (a_dtype == QS_BF16 && w_dtype == QS_F32 && c_dtype == QS_F32) GO(bf16, float, float);
#undef GO
    return qs_fail(QS_ERR_INVALID_INPUT, "linear: unsupported types A=%d W=%d C=%d", a_dtype, w_dtype, c_dtype);
}
