// True float32 matrix product C[M,N] = A[M,K] . W[N,K]^T with float32 FMA on the CUDA cores: no tensor cores, no TF32.  It
// carries every projection of the 32-bit path.  In every kernel here an output element is one chain of multiply-adds over
// K in ascending order, so its bits depend on K alone: not on M, not on the kernel that the sizes chose, and a token's result
// does not change with what else is in the batch.            (reference: cuBLAS, kernels/src/lib.rs:298-321)
//
//   tiles      outer products of 8 x 4 or 4 x 4 outputs a thread, both matrices through a ring of cp.async stages.  Bound by the
//              multiply-add pipe and by shared memory.  Plain fmaf, not fma.rn.f32x2: with three operands of 64 bits the
//              packed form stops at half the rate (a loop over registers: 68 TFLOP/s plain, 37 packed; the product of 2,048
//              rows, N 4,096, K 1,024 517 us packed, 394 plain).
//   few rows   (M <= 8) the weights streamed once, a lane a column and some rows.  Bound by the weights' bytes and, for
//              short rows of few columns, by the chain of K multiply-adds.
//
// Alone, before (one shape of 64 x 64 tiles, transposed element by element, two barriers every 16 elements of K) and now:
// N 4,096, K 1,024: 1 row 161 -> 15 us, 32 rows 161 -> 21, 128 rows 157 -> 38, 777 rows 320 -> 169, 2,048 rows 587 -> 385
// (45 TFLOP/s); N 1,024, K 2,048: 8 rows 297 -> 19, 777 rows 314 -> 120; N = K = 4,096: 8 rows 647 -> 49, 512 rows 877 -> 422.
#include "common.cuh"

namespace {

// PIECE bytes from global to shared memory, zeros where `live` is false
template <int PIECE>
__device__ __forceinline__ void copy_piece(float* to, const float* from, bool live) {
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(to);
    if (PIECE == 16) asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(at), "l"(from), "r"(live ? 16 : 0));
    else asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"(at), "l"(from), "r"(live ? 4 : 0));
}

// Rows of A and W lie in shared memory as they lie in memory, BK elements a row, with four floats between rows, so that the
// sixteen bytes that 8 neighbouring rows' readers take fall on 32 banks once.  A warp is 4 x 8 threads; a thread has the rows
// lane / 8 + 4 i and the columns lane % 8 + 8 j of its warp's part and reads four elements of K of each at a time.
// VEC: sixteen-byte copies (K a multiple of 4, both matrices on 16-byte boundaries), else four-byte ones.
template <int BM, int BN, int TM, int TN, int BK, int STAGES, int MIN_CTAS, bool VEC>
__global__ void __launch_bounds__((BM / TM) * (BN / TN), MIN_CTAS) gemm_f32_tiles_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                                        float* __restrict__ C, int M, int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / TN), WARPS_N = BN / (8 * TN), PITCH = BK + 4, STAGE = (BM + BN) * PITCH;
    constexpr int PIECE = VEC ? 4 : 1, PIECES = BK / PIECE;
    static_assert((BM + BN) * PIECES % THREADS == 0, "whole copies");
    extern __shared__ __align__(16) float ring[];
    pdl_launch_dependents();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tm = (warp / WARPS_N) * 4 * TM + (lane >> 3), tn = (warp % WARPS_N) * 8 * TN + (lane & 7);
    const int steps = (K + BK - 1) / BK;
    auto issue = [&](int step) {
        if (step < steps) {
            float* stage = ring + (step % STAGES) * STAGE;
#pragma unroll
            for (int i = 0; i < (BM + BN) * PIECES / THREADS; ++i) {
                const int idx = tid + i * THREADS, row = idx / PIECES, c = idx % PIECES * PIECE, k = step * BK + c;
                // rows beyond the last repeat it and are not stored
                const float* from = row < BM ? A + (size_t)min(m0 + row, M - 1) * K : W + (size_t)min(n0 + row - BM, N - 1) * K;
                copy_piece<4 * PIECE>(stage + row * PITCH + c, from + (k < K ? k : 0), k < K);
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.0f;
#pragma unroll 1
    for (int s = 0; s < STAGES - 1; ++s) issue(s);
#pragma unroll 1
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2));
        __syncthreads();                                     // the stage is there, and the one before it has been read
        issue(step + STAGES - 1);
        const float* a_s = ring + (step % STAGES) * STAGE + tm * PITCH;
        const float* w_s = ring + (step % STAGES) * STAGE + (BM + tn) * PITCH;
#pragma unroll
        for (int kk = 0; kk < BK; kk += 4) {
            float w[TN][4];
#pragma unroll
            for (int j = 0; j < TN; ++j) *reinterpret_cast<float4*>(w[j]) = *reinterpret_cast<const float4*>(w_s + 8 * j * PITCH + kk);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                float a[4];
                *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(a_s + 4 * i * PITCH + kk);
#pragma unroll
                for (int u = 0; u < 4; ++u)
#pragma unroll
                    for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[u], w[j][u], acc[i][j]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + tm + 4 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tn + 8 * j;
            if (n < N) C[(size_t)m * N + n] = acc[i][j];
        }
    }
}

// Up to 8 rows: a block has 16 columns over the whole of K (two warps of 8 columns, four lanes a column with R rows each), W
// and A come through a ring of stages of 128 elements of K.  K a multiple of 4, A and W on 16-byte boundaries.
constexpr int FEW_COLS = 16, FEW_K = 128, FEW_PITCH = FEW_K + 4, FEW_STAGES = 6, FEW_THREADS = 64;

template <int R>
__global__ void __launch_bounds__(FEW_THREADS) gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W,
                                                                  float* __restrict__ C, int M, int N, int K) {
    constexpr int ROWS = 4 * R, STAGE = (FEW_COLS + ROWS) * FEW_PITCH;
    extern __shared__ __align__(16) float ring[];
    pdl_launch_dependents();
    pdl_wait();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int n0 = blockIdx.x * FEW_COLS, steps = (K + FEW_K - 1) / FEW_K;
    auto issue = [&](int step) {
        if (step < steps) {
            float* stage = ring + (step % FEW_STAGES) * STAGE;
            const int k0 = step * FEW_K, live = min(FEW_K, K - k0) / 4;      // sixteen bytes a copy
            if (lane < live) {
                for (int r = warp; r < FEW_COLS + ROWS; r += FEW_THREADS / 32) {
                    // a column or row beyond the last repeats it and is not stored
                    const float* from = r < FEW_COLS ? W + (size_t)min(n0 + r, N - 1) * K : A + (size_t)min(r - FEW_COLS, M - 1) * K;
                    copy_piece<16>(stage + r * FEW_PITCH + 4 * lane, from + k0 + 4 * lane, true);
                }
            }
        }
        asm volatile("cp.async.commit_group;\n" ::);
    };
    for (int s = 0; s < FEW_STAGES - 1; ++s) issue(s);
    const int col = warp * 8 + (lane & 7), row = lane >> 3;                  // rows row, row + 4, ...
    float acc[R];
#pragma unroll
    for (int i = 0; i < R; ++i) acc[i] = 0.0f;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(FEW_STAGES - 2));
        __syncthreads();                                                     // the stage is there, and the one before it read
        issue(step + FEW_STAGES - 1);
        const float* stage = ring + (step % FEW_STAGES) * STAGE;
        const float* w = stage + col * FEW_PITCH;
        const float* a = stage + (FEW_COLS + row) * FEW_PITCH;
        const int live = min(FEW_K, K - step * FEW_K);
        // the chain of multiply-adds is short of work to hide a read behind: the next 16 elements are read ahead of it
        float4 wv[2][4], av[2][R][4];
        auto read = [&](int buffer, int k) {
#pragma unroll
            for (int u = 0; u < 4; ++u) {
                wv[buffer][u] = *reinterpret_cast<const float4*>(w + k + 4 * u);
#pragma unroll
                for (int i = 0; i < R; ++i) av[buffer][i][u] = *reinterpret_cast<const float4*>(a + 4 * i * FEW_PITCH + k + 4 * u);
            }
        };
        auto add = [&](float4 x, const float4 (&y)[R][4], int u) {
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(y[i][u].x, x.x, acc[i]);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(y[i][u].y, x.y, acc[i]);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(y[i][u].z, x.z, acc[i]);
#pragma unroll
            for (int i = 0; i < R; ++i) acc[i] = fmaf(y[i][u].w, x.w, acc[i]);
        };
        if (live == FEW_K) {
            read(0, 0);
#pragma unroll
            for (int k = 0; k < FEW_K; k += 16) {
                const int buffer = (k / 16) & 1;
                if (k + 16 < FEW_K) read(buffer ^ 1, k + 16);
#pragma unroll
                for (int u = 0; u < 4; ++u) add(wv[buffer][u], av[buffer], u);
            }
        } else {
            for (int k = 0; k < live; k += 4) {
                wv[0][0] = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
                for (int i = 0; i < R; ++i) av[0][i][0] = *reinterpret_cast<const float4*>(a + 4 * i * FEW_PITCH + k);
                add(wv[0][0], av[0], 0);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::);
    if (n0 + col >= N) return;
#pragma unroll
    for (int i = 0; i < R; ++i)
        if (row + 4 * i < M) C[(size_t)(row + 4 * i) * N + n0 + col] = acc[i];
}

template <int BM, int BN, int TM, int TN, int BK, int STAGES, int MIN_CTAS, bool VEC>
int launch_tiles(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    constexpr int SMEM = STAGES * (BM + BN) * (BK + 4) * (int)sizeof(float);
    static PerDevice configured;
    auto kernel = gemm_f32_tiles_kernel<BM, BN, TM, TN, BK, STAGES, MIN_CTAS, VEC>;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM);
    if (grid.y > 65535) return MRS_BAD_ARGUMENT;
    MRS_LAUNCH(kernel, grid, (BM / TM) * (BN / TN), SMEM, stream, A, W, C, M, N, K);
    MRS_RETURN_LAUNCH_STATUS();
}

template <bool VEC>
int launch_shape(int shape, const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    switch (shape) {
        case 0: return launch_tiles<64, 64, 8, 4, 16, 4, 4, VEC>(A, W, C, M, N, K, stream);
        case 1: return launch_tiles<32, 64, 4, 4, 32, 4, 4, VEC>(A, W, C, M, N, K, stream);
        case 2: return launch_tiles<32, 32, 4, 4, 32, 6, 4, VEC>(A, W, C, M, N, K, stream);
    }
    return MRS_BAD_ARGUMENT;
}

template <int R>
int launch_few(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    constexpr int SMEM = FEW_STAGES * (FEW_COLS + 4 * R) * FEW_PITCH * (int)sizeof(float);
    static PerDevice configured;
    if (!configured.get()) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM);
        if (e != cudaSuccess) return (int)e;
        configured.set(1);
    }
    MRS_LAUNCH(gemm_f32_few_kernel<R>, (N + FEW_COLS - 1) / FEW_COLS, FEW_THREADS, SMEM, stream, A, W, C, M, N, K);
    MRS_RETURN_LAUNCH_STATUS();
}

}  // namespace

MRS_EXPORT int mrs_gemm_f32(const float* A, const float* W, float* C, int M, int N, int K, void* stream) {
    if (M <= 0 || N <= 0) return 0;
    if (K <= 0) return MRS_BAD_ARGUMENT;
    const bool vec = K % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (M <= 8 && vec) return M <= 4 ? launch_few<1>(A, W, C, M, N, K, stream) : launch_few<2>(A, W, C, M, N, K, stream);
    // A shape's time over q tiles an SM, in microseconds at K = 1,024, is a line: measured alone at N = 1,024 to 6,144,
    // M = 17 to 2,048, q = 1 to 55 (within a fifth of it nearly everywhere).  The wide tiles win when every SM has many
    // (2,048 rows, N 4,096: 384, 418 and 457 us for the three shapes; 64 rows: 40, 30, 34; 32 rows of N = 1,024: 37, 22, 18).
    // A grid's second dimension ends at 65,535 tiles of rows: beyond what the low tiles cover, the high ones take the product.
    const int bm[3] = {64, 32, 32}, bn[3] = {64, 64, 32}, sms = mrs_sm_count();
    const double first[3] = {45.0, 19.0, 12.0}, each[3] = {24.0, 14.3, 8.6};
    double best = 0.0;
    int shape = 0;
    for (int i = 0; i < 3; ++i) {
        const long long rows = ((long long)M + bm[i] - 1) / bm[i], tiles = rows * ((N + bn[i] - 1) / bn[i]);
        const double time = first[i] + each[i] * (double)((tiles + sms - 1) / sms);
        if (i == 0 || (time < best && rows <= 65535)) best = time, shape = i;
    }
    return vec ? launch_shape<true>(shape, A, W, C, M, N, K, stream) : launch_shape<false>(shape, A, W, C, M, N, K, stream);
}
