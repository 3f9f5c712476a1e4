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
#include "common.cuh"

#define GP_BM 64
#define GP_BN 64
#define GP_BK 16
#define GP_RUN 256    // products summed in order before their sum joins the total; a multiple of GP_BK

// ------------------------------------------------------------------------------------------------ 32-bit operands
// A tile of 8 TM x 8 TN sums by groups of 64 threads (8 x 8, a thread TM x TN sums): every group forms whole runs of GP_RUN
// products, as many runs at once as there are groups, and their sums are added in the runs' order from shared memory. What runs
// of one tile share is only that addition, so a block is 2 to 16 warps of independent work on a tile whatever K is, and the
// order of the sums is the one above. Operands go to shared memory as they lie (rows of GP_BK values, by asynchronous
// copies, two stages a group) and are read four values of k at a time: (TM + TN) 16-byte reads for 4 TM TN multiply-adds, so
// 64 x 64 is bound by the multiply-adds and the smaller tiles by shared memory; those are for products whose 64 x 64 tiles
// leave SMs idle. 2,048 x 2,048 x 2,048: 31 TFLOP/s; 213 x 2,560 x 1,536: 25 (64 x 64 tiles of 256 threads, run after run: about 7).
#define GP_PITCH (GP_BK + 4)

__device__ __forceinline__ void gp_copy(float* dst, const float* src, int bytes, bool in) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    const int n = in ? bytes : 0;           // nothing is read from outside; zeros instead
    if (bytes == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}

template <int TM, int TN> struct RunTile {
    static constexpr int BM = 8 * TM, BN = 8 * TN, STAGE = (BM + BN) * GP_PITCH;      // floats a stage
    static constexpr size_t smem(int groups) { return (size_t)(groups * 2 * STAGE + BM * BN) * sizeof(float); }
};

template <int TM, int TN>
__global__ void __launch_bounds__(512)
gemm_runs_kernel(float* __restrict__ C, const float* __restrict__ A, const float* __restrict__ W, int M, int N, int K,
                 long long lda, long long ldw, long long ldc, int vec) {
    using T = RunTile<TM, TN>;
    constexpr int BM = T::BM, BN = T::BN;
    static_assert(BM * BN <= 2 * T::STAGE, "a group's sums take the place of its stages");
    extern __shared__ __align__(16) float gp_smem[];
    const int groups = blockDim.x / 64, g = threadIdx.x / 64, tid = threadIdx.x & 63, tx = tid & 7, ty = tid >> 3;
    float* mine = gp_smem + g * 2 * T::STAGE;
    float* total = gp_smem + groups * 2 * T::STAGE;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN, n_runs = (K + GP_RUN - 1) / GP_RUN;
    pdl_trigger();
    pdl_wait();
    for (int i = threadIdx.x; i < BM * BN; i += blockDim.x) total[i] = 0.f;
    auto group_sync = [&]() { asm volatile("bar.sync %0, 64;" ::"r"(g + 1) : "memory"); };
    auto issue = [&](int stage, int k0) {
        float* dst = mine + stage * T::STAGE;
        const int shift = vec ? 2 : 4, width = vec ? 4 : 1;          // copies of a row: 4 of four values, or 16 of one
        for (int i = tid; i < (BM + BN) << shift; i += 64) {
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
                        const float4 a = *reinterpret_cast<const float4*>(as + i * 8 * GP_PITCH + kk);
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
                for (int j = 0; j < TN; ++j) mine[(ty + 8 * i) * BN + tx + 8 * j] = acc[i][j];
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

template <int TM, int TN>
static int run_tiles(float* C, const float* A, const float* W, int M, int N, int K, long long lda, long long ldw, long long ldc,
                     int groups, int vec, cudaStream_t stream) {
    using T = RunTile<TM, TN>;
    const dim3 grid((unsigned)((N + T::BN - 1) / T::BN), (unsigned)((M + T::BM - 1) / T::BM));
    if (grid.y > 65535) return CELLM_ERR_SIZE;
    cudaError_t e = cudaFuncSetAttribute(gemm_runs_kernel<TM, TN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)T::smem(8));
    if (e != cudaSuccess) return (int)e;
    CELLM_RUN((gemm_runs_kernel<TM, TN>), grid, groups * 64, T::smem(groups), stream, C, A, W, M, N, K, lda, ldw, ldc, vec);
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
        // The tile whose waves over the SMs take least. Microseconds of K = 1,536 measured for one tile an SM and for each
        // wave of several (the smaller tiles share an SM then): with 213 x 2,560 sums 64 x 64 takes 125 us, 32 x 64 68, 32 x 32
        // 87, 16 x 32 96; with 16 x 1,536 they take 63, 34, 22 and 18; with 2,048 x 2,048 (K 2,048) 545, 577, 723 and 836.
        static const struct { int bm, bn; double alone, wave; } tile[4] = {{64, 64, 62.8, 60.}, {32, 64, 34.4, 33.}, {32, 32, 22.4, 21.}, {16, 32, 18., 12.}};
        int best = 0;
        double least = 0;
        for (int i = 0; i < 4; ++i) {
            if (i > 0 && (M + tile[i].bm - 1) / tile[i].bm > 65535) break;      // as many rows as 64 x 64 tiles take, whatever their number
            const long long tiles = (long long)((M + tile[i].bm - 1) / tile[i].bm) * ((N + tile[i].bn - 1) / tile[i].bn), waves = (tiles + 147) / 148;
            const double cost = waves == 1 ? tile[i].alone : (double)waves * tile[i].wave;
            if (i == 0 || cost < least) best = i, least = cost;
        }
#define RUNS(TM, TN) return run_tiles<TM, TN>((float*)C, (const float*)A, (const float*)W, M, N, K, lda, ldw, ldc, groups, vec, stream)
        if (best == 0) RUNS(8, 8);
        if (best == 1) RUNS(4, 8);
        if (best == 2) RUNS(4, 4);
        RUNS(2, 4);
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
