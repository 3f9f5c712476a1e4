// Plain matrix product on the CUDA cores: C[M,N] = A[M,K] . W[N,K]^T with
// 32-bit multiply-add and 32-bit sums, no tensor cores and no reduced-precision
// mode. Every element of C is summed over k in runs of GP_RUN consecutive
// products, each run in order, and the runs' sums are added in order: the
// rounding of a sum of K terms then grows like sqrt(GP_RUN) + sqrt(K / GP_RUN)
// units instead of sqrt(K), and the order depends on K alone, whatever the tile
// an element falls in, so a row's result does not depend on the other rows of
// the batch. It is the product of the 32-bit path and the reference for the tensor
// core kernels (the reference's own linear is a scalar loop over k,
// crates/cellm-model/src/lfm.rs:970-978).
//
// 32-bit operands: the runs of a tile are summed by different groups of threads at once (gemm_runs_kernel); short products of
// many tiles, rows off the 16-byte border and bfloat16 operands (products the tensor-core kernels do not take) by one group, run
// after run. Both give the same sums.
#include <algorithm>
#include <cmath>

#include "common.cuh"

#define GP_BM 64
#define GP_BN 64
#define GP_BK 16
#define GP_RUN 256    // products summed in order before their sum joins the total; a multiple of GP_BK

// ------------------------------------------------------------------------------------------------ 32-bit operands
// A tile of LY TM x 8 TN sums by groups of 8 LY threads (64, or a warp; a thread TM x TN sums): every group forms whole runs of GP_RUN
// products, as many runs at once as there are groups, and their sums are added in the runs' order from shared memory. What runs
// of one tile share is only that addition, so a block is 2 to 16 warps of independent work on a tile whatever K is, and the
// order of the sums is the one above. Operands go to shared memory as they lie (rows of GP_BK values, by asynchronous
// copies, two stages a group) and are read four values of k at a time: (TM + TN) 16-byte reads for 4 TM TN multiply-adds, so
// 64 x 64 is bound by the multiply-adds and the smaller tiles by shared memory; those are for products whose 64 x 64 tiles
// leave SMs idle. Single warps have no barrier and a quarter of a 64-thread tile's rows: blocks of few registers that share an SM and
// fill it evenly. 2,048 x 2,048 x 2,048: 37 TFLOP/s; 261 x 2,560 x 1,536: 27 (in tiles of 32 x 64 by 64 threads 20).
#define GP_PITCH (GP_BK + 4)

__device__ __forceinline__ void gp_copy(float* dst, const float* src, int bytes, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = in ? bytes : 0;           // nothing is read from outside; zeros instead
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int TM, int TN, int LY> struct RunTile {
    static constexpr int BM = LY * TM, BN = 8 * TN, STAGE = (BM + BN) * GP_PITCH;      // floats a stage
    static constexpr size_t smem(int groups) { return (size_t)(groups * 2 * STAGE + BM * BN) * sizeof(float); }
};

template <int TM, int TN, int LY>
__global__ void __launch_bounds__(LY * 64)
gemm_runs_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, int vec) {
    using T = RunTile<TM, TN, LY>;
    constexpr int BM = T::BM, BN = T::BN, GT = 8 * LY;
    static_assert(BM % (GT / 4) == 0 && BN % (GT / 4) == 0, "a thread's copies are of whole tiles");
    static_assert(BM * BN <= 2 * T::STAGE, "a group's sums take the place of its stages");
    extern __shared__ __align__(16) float gp_smem[];
    const int groups = blockDim.x / GT, g = threadIdx.x / GT, tid = threadIdx.x % GT;
    // a 16-byte read of shared memory costs half where neighbouring lanes read the same: one operand's in either form
    const int tx = LY == 4 ? (tid >> 1) & 7 : tid & 7, ty = LY == 4 ? (tid & 1) | (tid >> 4) << 1 : tid >> 3;
    float* mine = gp_smem + g * 2 * T::STAGE;
    float* total = gp_smem + groups * 2 * T::STAGE;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, n_runs = (K + GP_RUN - 1) / GP_RUN;
    pdl_trigger();
    pdl_wait();
    for (int i = threadIdx.x; i < BM * BN; i += blockDim.x) total[i] = 0.f;
    auto group_sync = [&]() { if constexpr (GT == 32) __syncwarp(); else asm volatile("bar.sync %0, %1;" ::"r"(g + 1), "n"(GT) : "memory"); };
    auto issue = [&](int stage, int k0) {
        float* dst = mine + stage * T::STAGE;
        if (vec) {          // a thread's copies: the same four values of k in rows GT / 4 apart
            const int kk = (tid & 3) * 4, r0 = tid >> 2, gk = k0 + kk;
            const float *a = A + (size_t)(m0 + r0) * lda + gk, *w = W + (size_t)(n0 + r0) * ldw + gk;
            float* to = dst + r0 * GP_PITCH + kk;
#pragma unroll
            for (int i = 0; i < BM; i += GT / 4) {
                const bool in = m0 + r0 + i < M && gk < K;
                gp_copy(to + i * GP_PITCH, in ? a + (size_t)i * lda : A, 16, in);
            }
#pragma unroll
            for (int i = 0; i < BN; i += GT / 4) {
                const bool in = n0 + r0 + i < N && gk < K;
                gp_copy(to + (BM + i) * GP_PITCH, in ? w + (size_t)i * ldw : W, 16, in);
            }
            return;
        }
        constexpr int shift = 4, width = 1;          // a row's copies: 16 of one value
        for (int i = tid; i < (BM + BN) << shift; i += GT) {
            const int r = i >> shift, kk = (i & ((1 << shift) - 1)) * width, gk = k0 + kk;
            const bool w_row = r >= BM;
            const int row = w_row ? n0 + r - BM : m0 + r;
            const bool in = row < (w_row ? N : M) && gk < K;
            const float* base = w_row ? W : A;
            gp_copy(dst + r * GP_PITCH + kk, in ? base + (size_t)row * (w_row ? ldw : lda) + gk : base, 4 * width, in);
        }
    };
    for (int r0 = 0; r0 < n_runs; r0 += groups) {
        const int run = r0 + g;
        if (run < n_runs) {
            float acc[TM][TN];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
            const int k_begin = run * GP_RUN, steps = (min(GP_RUN, K - k_begin) + GP_BK - 1) / GP_BK;
            issue(0, k_begin);
            asm volatile("cp.async.commit_group;" ::: "memory");
            for (int s = 0; s < steps; ++s) {
                if (s + 1 < steps) issue((s + 1) & 1, k_begin + (s + 1) * GP_BK);
                asm volatile("cp.async.commit_group;" ::: "memory");
                asm volatile("cp.async.wait_group 1;" ::: "memory");
                group_sync();
                const float* as = mine + (s & 1) * T::STAGE + ty * GP_PITCH;
                const float* ws = mine + (s & 1) * T::STAGE + (BM + tx) * GP_PITCH;
#pragma unroll
                for (int kk = 0; kk < GP_BK; kk += 4) {
                    float4 w[TN];
#pragma unroll
                    for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + j * 8 * GP_PITCH + kk);
#pragma unroll
                    for (int i = 0; i < TM; ++i) {
                        const float4 a = *reinterpret_cast<const float4*>(as + i * LY * GP_PITCH + kk);
#pragma unroll
                        for (int j = 0; j < TN; ++j) {
                            acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
                            acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
                            acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
                            acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
                        }
                    }
                }
                group_sync();
            }
            asm volatile("cp.async.wait_group 0;" ::: "memory");
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) mine[(ty + LY * i) * BN + tx + 8 * j] = acc[i][j];
        }
        __syncthreads();
        for (int i = threadIdx.x; i < BM * BN; i += blockDim.x) {
            float sum = total[i];
            for (int r = 0; r < groups && r0 + r < n_runs; ++r) sum += gp_smem[r * 2 * T::STAGE + i];
            total[i] = sum;
        }
        __syncthreads();
    }
    for (int i = threadIdx.x; i < BM * BN; i += blockDim.x) {
        const int gm = m0 + i / BN, gn = n0 + i % BN;
        if (gm < M && gn < N) C[(size_t)gm * ldc + gn] = total[i];
    }
}

template <int TM, int TN, int LY>
static int run_tiles(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldw, long long ldc,
                     int groups, int vec, cudaStream_t stream) {
    using T = RunTile<TM, TN, LY>;
    const dim3 grid((unsigned)((N + T::BN - 1) / T::BN), (unsigned)((M + T::BM - 1) / T::BM));
    if (grid.y > 65535) return CELLM_ERR_SIZE;
    cudaError_t e = cudaFuncSetAttribute(gemm_runs_kernel<TM, TN, LY>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem(8));
    if (e != cudaSuccess) return (int)e;
    CELLM_RUN((gemm_runs_kernel<TM, TN, LY>), grid, groups * 8 * LY, T::smem(groups), stream, C, A, W, M, N, K, lda, ldw, ldc, vec);
    return CELLM_OK;
}

// ------------------------------------------------------------------------------------------------ run after run
template <typename TI, typename TO>
__global__ void __launch_bounds__(256)
gemm_plain_kernel(TO* __restrict__ C, const TI* __restrict__ A, const TI* __restrict__ W, int M, int N,
                  int K, long long lda, long long ldw, long long ldc) {
    __shared__ float As[GP_BK][GP_BM + 4];
    __shared__ float Ws[GP_BK][GP_BN + 4];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x;
    const int tx = tid & 15, ty = tid >> 4;
    const int m0 = blockIdx.y * GP_BM, n0 = blockIdx.x * GP_BN;
    float acc[4][4], total[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = total[i][j] = 0.f;
    for (int k0 = 0; k0 < K; k0 += GP_BK) {
        if (k0 && k0 % GP_RUN == 0) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) { total[i][j] += acc[i][j]; acc[i][j] = 0.f; }
        }
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const int idx = tid + r * 256;
            const int row = idx >> 4, kk = idx & 15;
            const int gm = m0 + row, gn = n0 + row, gk = k0 + kk;
            As[kk][row] = (gm < M && gk < K) ? to_float(A[(size_t)gm * lda + gk]) : 0.f;
            Ws[kk][row] = (gn < N && gk < K) ? to_float(W[(size_t)gn * ldw + gk]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < GP_BK; ++kk) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gm = m0 + ty * 4 + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gn = n0 + tx * 4 + j;
            if (gn < N) C[(size_t)gm * ldc + gn] = from_float<TO>(total[i][j] + acc[i][j]);
        }
    }
}

// A: [M, K] (row stride lda), W: [N, K] (row stride ldw), both of in_dtype;
// C: [M, N] (row stride ldc) of out_dtype.
CELLM_API int cellm_gemm_plain(void* C, const void* A, const void* W, int M, int N, int K, long long lda,
                               long long ldw, long long ldc, int in_dtype, int out_dtype,
                               cudaStream_t stream) {
    if (M <= 0 || N <= 0) return CELLM_OK;
    if (K <= 0) return CELLM_ERR_SIZE;
    // 32-bit operands go to the groups of threads from two runs of products on, and below where the 64 x 64 tiles are few; rows off
    // the 16-byte border (copied value by value) only where those are very few. Elsewhere the tile's 256 threads of the other kernel
    // hide more. Its time over the groups', products of 1 to 2,048 rows by 512 to 8,192 columns: K 512 to 1,536 0.97 to 5.2; K 32 to
    // 300 0.98 to 2.5 where the line says groups, 0.46 to 1.02 where it does not (2,048 x 2,048 x 64: 27 against 40 us); K 513 1.65
    // to 1.8 and 0.56 to 1.0. The sums are the same bits either way.
    const int vec = K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    const long long tiles64 = (long long)((M + GP_BM - 1) / GP_BM) * ((N + GP_BN - 1) / GP_BN);
    const long long few = M <= 16 ? 32 : vec ? (K / 4 < 32 ? K / 4 : 32) : 8;
    if (in_dtype == CELLM_F32 && out_dtype == CELLM_F32 && ((vec && K >= 2 * GP_RUN) || tiles64 <= few)) {
        const int n_runs = (K + GP_RUN - 1) / GP_RUN, rounds = (n_runs + 7) / 8, groups = (n_runs + rounds - 1) / rounds;
        // The tile whose waves over the SMs take least: measured microseconds of one tile an SM (`alone`), else of each wave, behind
        // `first` and no less than `least`; `step` waves start together (1: a block fills an SM; 2: two share it; 0: blocks so small
        // that their waves melt together).
        struct Tile { int bm, bn; double alone, wave, first, least; int step; };
        // Five groups and more, K = 1,536. 213 x 2,560 sums take 108 us in tiles of 64 x 64, 63 of 32 x 64, 77 of 32 x 32, 85 of
        // 16 x 32, 64 and 63 of those by single warps; 261 x 2,560 111, 91, 95, 105, 92, 77; 16 x 1,536 55, 31, 20, 14, 21, 16;
        // 2,048 x 2,048 (K 2,048) 468, 540, 657, 859, 519, 560.
        static const Tile long_k[6] = {{64, 64, 58., 52., 0., 0., 1}, {32, 64, 32., 30., 0., 0., 1}, {32, 32, 20.5, 19.3, 0., 0., 1},
                                       {16, 32, 14.3, 11.5, 0., 0., 1}, {32, 32, 25., 14.3, 10., 33., 0}, {16, 32, 16.5, 7.65, 5., 33., 0}};
        // Four, K = 1,024. 261 x 2,560: 74, 73, 68, 69, 58, 51 us; 400 x 1,536 74, 64, 66, 62, 57, 47; 64 x 2,560 44, 34, 25, 24, 31, 29;
        // 700 x 2,560 113, 116, 139, 161, 114, 117; 2,048 x 1,536 214, 208, 244, 277, 196, 197.
        static const Tile four[6] = {{64, 64, 44., 36., 0., 0., 1}, {32, 64, 26., 20.5, 0., 0., 1}, {32, 32, 18., 11.6, 12., 0., 0},
                                     {16, 32, 14., 6.6, 8., 21., 0}, {32, 32, 23., 9.1, 9., 29., 0}, {16, 32, 13., 4.6, 8., 28., 0}};
        // Three, K = 768. 261 x 2,560: 57, 60, 48, 53, 40, 43 us; 400 x 1,536 57, 59, 44, 48, 40, 39; 100 x 1,536 41, 28, 25, 23, 28, 25;
        // 2,048 x 1,536 164, 173, 166, 210, 154, 151 (tiles of 32 x 32 by single warps win nowhere by more than 3 us, and lose 10 where
        // nearly six an SM meet).
        static const Tile three[6] = {{64, 64, 40., 27.4, 0., 0., 2}, {32, 64, 28., 14.8, 0., 0., 2}, {32, 32, 16.3, 8., 8., 24.6, 0},
                                      {16, 32, 10.6, 5.1, 5., 17.7, 0}, {0}, {16, 32, 12., 3.3, 15., 15.6, 0}};
        // Fewer (single warps are too few of them then), and rows off the 16-byte border.
        static const Tile short_k[6] = {{64, 64, 62.8, 60., 0., 0., 1}, {32, 64, 34.4, 33., 0., 0., 1}, {32, 32, 22.4, 21., 0., 0., 1},
                                        {16, 32, 18., 12., 0., 0., 1}, {0}, {0}};
        const Tile* const tiles = !vec || groups < 3 ? short_k : groups == 3 ? three : groups == 4 ? four : long_k;
        int best = 0;
        double least = 0;
        for (int i = 0; i < 6; ++i) {
            const Tile& t = tiles[i];
            if (!t.bm || (i > 0 && (M + t.bm - 1) / t.bm > 65535)) continue;      // as many rows as 64 x 64 tiles take, whatever their number
            const double waves = (double)((long long)((M + t.bm - 1) / t.bm) * ((N + t.bn - 1) / t.bn)) / 148.;
            double cost = t.alone;
            if (waves > 1.) cost = std::max(t.least, t.first + (t.step ? ceil(waves / t.step) * t.step : waves) * t.wave);
            else if (tiles == long_k && i == 3 && waves * 148. > 64.) cost = 19.6;          // (more than 64 of these wait for memory together)
            if (i == 0 || cost < least) best = i, least = cost;
        }
#define RUNS(TM, TN, LY) return run_tiles<TM, TN, LY>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, groups, vec, stream)
        if (best == 0) RUNS(8, 8, 8);
        if (best == 1) RUNS(4, 8, 8);
        if (best == 2) RUNS(4, 4, 8);
        if (best == 3) RUNS(2, 4, 8);
        if (best == 4) RUNS(8, 4, 4);
        RUNS(4, 4, 4);
#undef RUNS
    }
    const dim3 grid((unsigned)((N + GP_BN - 1) / GP_BN), (unsigned)((M + GP_BM - 1) / GP_BM));
    if (grid.y > 65535) return CELLM_ERR_SIZE;
#define LAUNCH(TI, TO) \
    CELLM_RUN((gemm_plain_kernel<TI, TO>), grid, 256, 0, stream, (TO*)C, (const TI*)A, (const TI*)W, M, N, K, lda, ldw, ldc)
    if (in_dtype == CELLM_F32 && out_dtype == CELLM_F32) LAUNCH(float, float);
    else if (in_dtype == CELLM_BF16 && out_dtype == CELLM_BF16) LAUNCH(__nv_bfloat16, __nv_bfloat16);
    else if (in_dtype == CELLM_BF16 && out_dtype == CELLM_F32) LAUNCH(__nv_bfloat16, float);
    else return CELLM_ERR_DTYPE;
#undef LAUNCH
    return CELLM_OK;
}
