// True float32 matrix product on the CUDA cores (FMA; no tensor cores, no TF32):
//   C[M, N] = A[M, K] . W[N, K]^T        (weights as stored by HF: [out, in])
// It is the 32-bit path of every projection and of the LM head.  Each output
// element is one thread's running sum over k = 0 .. K-1 in that order, so a
// row's result does not depend on M: the same token gives the same bits
// whatever else is in the batch.
// The reference multiplies x[B,S,in] by a weight kept as [in,out]
// (crates/ai-engine-runtime/src/arch/linear.rs:106-123); the product is the same.
#include "common.cuh"

#define BM 64
#define BN 64
#define BK 16

template <typename AT, typename WT, typename OT>
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const AT* __restrict__ A, const WT* __restrict__ W, OT* __restrict__ C,
                const int* __restrict__ a_rows, const int* __restrict__ tile_w, int M, int N, int K, int lda,
                int ldc, long long a_bs, long long w_bs, long long c_bs) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    // a batch of products (blockIdx.z), or one weight per tile of rows (tile_w: -1 = the tile is empty)
    A += (long long)blockIdx.z * a_bs;
    C += (long long)blockIdx.z * c_bs;
    if (tile_w) {
        const int e = tile_w[blockIdx.y];
        if (e < 0) return;
        W += (long long)e * w_bs;
    } else {
        W += (long long)blockIdx.z * w_bs;
    }
    const int tm = (tid / 16) * 4, tn = (tid % 16) * 4;
    float acc[4][4];
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0.f;

    // loader mapping: 64 rows x 16 k per tile, 256 threads -> 4 consecutive k each
    const int lr = tid / 4, lk = (tid % 4) * 4;
    const int am = m0 + lr, wn = n0 + lr;
    const AT* arow = nullptr;
    if (am < M) {
        const int r = a_rows ? a_rows[am] : am;
        if (r >= 0) arow = A + (size_t)r * lda;
    }
    const WT* wrow = wn < N ? W + (size_t)wn * K : nullptr;

    for (int k0 = 0; k0 < K; k0 += BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            As[lk + j][lr] = (arow && k < K) ? to_f32<AT>(arow[k]) : 0.f;
            Ws[lk + j][lr] = (wrow && k < K) ? to_f32<WT>(wrow[k]) : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < BK; ++k) {
            float a[4], w[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[k][tm + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) w[j] = Ws[k][tn + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int m = m0 + tm + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int n = n0 + tn + j;
            if (n < N) C[(size_t)m * ldc + n] = from_f32<OT>(acc[i][j]);
        }
    }
}

template <typename AT, typename WT>
static int gemm_f32_go(const void* A, const void* W, void* C, int c_dtype, const int* a_rows, const int* tile_w,
                       int M, int N, int K, int lda, int ldc, int batch, long long a_bs, long long w_bs,
                       long long c_bs, cudaStream_t stream) {
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    if (grid.y > 65535 || batch > 65535) return AIE_UNSUPPORTED;
    if (c_dtype == AIE_F32)
        gemm_f32_kernel<AT, WT, float><<<grid, 256, 0, stream>>>((const AT*)A, (const WT*)W, (float*)C, a_rows, tile_w,
                                                                 M, N, K, lda, ldc, a_bs, w_bs, c_bs);
    else if (c_dtype == AIE_BF16)
        gemm_f32_kernel<AT, WT, bf16><<<grid, 256, 0, stream>>>((const AT*)A, (const WT*)W, (bf16*)C, a_rows, tile_w,
                                                                M, N, K, lda, ldc, a_bs, w_bs, c_bs);
    else
        return AIE_BAD_ARG;
    AIE_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The same product for float32 operands whose rows start on 16 bytes: blocks of 64 x 64 outputs, a thread 8 x 4 of them (a
// warp's lanes lie 4 x 8 over its quarter), tiles of 64 k brought by cp.async into two stages, k innermost as in memory
// (rows 68 floats apart: the eight rows that lanes read at a time fall on different banks).  Each output is still one
// thread's sum over k in order: bits do not depend on the tile.  Warps whose rows all lie behind M only help loading.
// Bound by what shared memory hands to registers (12 floats a thread for 32 multiply-adds: two thirds of the FMA rate)
// and, on small grids, by latency.  513 tokens, us, before -> now: 2,048 x 2,048 213 -> 123; 3,072 x 2,048 305 -> 174;
// 2,048 x 8,192 878 -> 461; 16,384 x 2,048 1,518 -> 881 (39 TFLOP/s).  Tiles of 64 x 128 and 128 x 128 with 8 x 8 or
// 16 x 8 a thread were within 4 % on the largest grids and 15 to 100 % slower on the others, tiles of 16 and 32 k
// 33 and 3 % slower in sum.
#define GT_M 64
#define GT_N 64
#define GT_K 64
#define GT_LD (GT_K + 4)
#define GT_STAGES 2
#define GT_THREADS 128
#define GT_TM 8
#define GT_TN 4

template <typename OT>
__global__ void __launch_bounds__(GT_THREADS, 3)
gemm_f32_tiled_kernel(const float* __restrict__ A, const float* __restrict__ W, OT* __restrict__ C,
                      const int* __restrict__ a_rows, const int* __restrict__ tile_w, int M, int N, int K, int lda, int ldc,
                      long long a_bs, long long w_bs, long long c_bs) {
    constexpr int ROW = GT_K / 4, PIECES = (GT_M + GT_N) * ROW / GT_THREADS, STEP = GT_THREADS / ROW, STAGE = (GT_M + GT_N) * GT_LD;
    extern __shared__ __align__(16) float gt_sm[];
    const int tid = threadIdx.x, lane = tid & 31, wm = tid >> 6, wn = (tid >> 5) & 1;
    const int m0 = blockIdx.y * GT_M, n0 = blockIdx.x * GT_N;
    A += (long long)blockIdx.z * a_bs;
    C += (long long)blockIdx.z * c_bs;
    if (tile_w) {
        const int e = tile_w[blockIdx.y];
        if (e < 0) return;
        W += (long long)e * w_bs;
    } else {
        W += (long long)blockIdx.z * w_bs;
    }
    // a thread's pieces of a tile: 16 bytes at column k4 of every STEP-th row, GT_M rows of A, then those of W
    const int row0 = tid / ROW, k4 = (tid % ROW) * 4;
    int arow[GT_M / STEP];                          // -1: a row of zeros
#pragma unroll
    for (int i = 0; i < GT_M / STEP; ++i) {
        const int m = m0 + row0 + i * STEP;
        arow[i] = m < M ? (a_rows ? a_rows[m] : m) : -1;
    }
    const int blocks = (K + GT_K - 1) / GT_K;
    auto fetch = [&](int kb) {
        if (kb < blocks) {
            const unsigned dst = (unsigned)__cvta_generic_to_shared(gt_sm + (kb % GT_STAGES) * STAGE + row0 * GT_LD + k4);
            const int k = kb * GT_K + k4;
#pragma unroll
            for (int i = 0; i < PIECES; ++i) {
                const float* src = W;
                bool ok = k < K;
                if (i < GT_M / STEP) {
                    ok = ok && arow[i < GT_M / STEP ? i : 0] >= 0;
                    if (ok) src = A + (size_t)arow[i < GT_M / STEP ? i : 0] * lda + k;
                } else {
                    const int n = n0 + row0 + (i - GT_M / STEP) * STEP;
                    ok = ok && n < N;
                    if (ok) src = W + (size_t)n * K + k;
                }
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(dst + i * STEP * GT_LD * 4), "l"(src),
                             "r"(ok ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float acc[GT_TM][GT_TN];
#pragma unroll
    for (int i = 0; i < GT_TM; ++i)
#pragma unroll
        for (int j = 0; j < GT_TN; ++j) acc[i][j] = 0.f;
    const int lm = wm * 4 * GT_TM + (lane >> 3), ln = wn * 8 * GT_TN + (lane & 7);        // rows lm + 4 i, columns ln + 8 j
    const bool works = m0 + wm * 4 * GT_TM < M;
#pragma unroll
    for (int s = 0; s < GT_STAGES - 1; ++s) fetch(s);
#pragma unroll 1
    for (int kb = 0; kb < blocks; ++kb) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(GT_STAGES - 2) : "memory");
        __syncthreads();
        fetch(kb + GT_STAGES - 1);
        if (!works) continue;
        const float* as = gt_sm + (kb % GT_STAGES) * STAGE + lm * GT_LD;
        const float* ws = gt_sm + (kb % GT_STAGES) * STAGE + (GT_M + ln) * GT_LD;
#pragma unroll 2
        for (int k = 0; k < GT_K; k += 4) {
            float4 a[GT_TM], w[GT_TN];
#pragma unroll
            for (int i = 0; i < GT_TM; ++i) a[i] = *reinterpret_cast<const float4*>(as + 4 * i * GT_LD + k);
#pragma unroll
            for (int j = 0; j < GT_TN; ++j) w[j] = *reinterpret_cast<const float4*>(ws + 8 * j * GT_LD + k);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int i = 0; i < GT_TM; ++i)
#pragma unroll
                    for (int j = 0; j < GT_TN; ++j)
                        acc[i][j] = x == 0 ? fmaf(a[i].x, w[j].x, acc[i][j]) : x == 1 ? fmaf(a[i].y, w[j].y, acc[i][j])
                                  : x == 2 ? fmaf(a[i].z, w[j].z, acc[i][j]) : fmaf(a[i].w, w[j].w, acc[i][j]);
        }
    }
#pragma unroll
    for (int i = 0; i < GT_TM; ++i) {
        const int m = m0 + lm + 4 * i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < GT_TN; ++j) {
            const int n = n0 + ln + 8 * j;
            if (n < N) C[(size_t)m * ldc + n] = from_f32<OT>(acc[i][j]);
        }
    }
}

template <typename OT>
static int gemm_f32_tiled(const float* A, const float* W, OT* C, const int* a_rows, const int* tile_w, int M, int N, int K,
                          int lda, int ldc, int batch, long long a_bs, long long w_bs, long long c_bs, cudaStream_t stream) {
    constexpr int smem = GT_STAGES * (GT_M + GT_N) * GT_LD * 4;
    dim3 grid((N + GT_N - 1) / GT_N, (M + GT_M - 1) / GT_M, batch);
    if (grid.y > 65535 || batch > 65535) return AIE_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_tiled_kernel<OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    gemm_f32_tiled_kernel<OT><<<grid, GT_THREADS, smem, stream>>>(A, W, C, a_rows, tile_w, M, N, K, lda, ldc, a_bs, w_bs, c_bs);
    AIE_LAUNCH_CHECK();
}

// The general form.  A [M, lda] (float32 or bfloat16, widened on load), W [N, K], C [M, ldc] (float32 or
// bfloat16, rounded once at the store).  a_rows (optional): row m of the product reads A[a_rows[m]] (a
// negative entry reads zeros).  batch > 1: `batch` independent products whose operands lie a_bs / w_bs / c_bs
// elements apart (per-head projections).  tile_w (optional, batch == 1): rows 64 i .. 64 i + 63 of the product
// use the weight W + tile_w[i] * w_bs (rows grouped by expert; -1 skips the tile).
extern "C" int aie_gemm_f32_ex(const void* A, int a_dtype, const void* W, int w_dtype, void* C, int c_dtype,
                               const int* a_rows, const int* tile_w, int M, int N, int K, int lda, int ldc,
                               int batch, long long a_bs, long long w_bs, long long c_bs, cudaStream_t stream) {
    if (M <= 0 || N <= 0 || batch <= 0) return 0;
    if (K <= 0 || (tile_w && batch != 1)) return AIE_BAD_ARG;
    if (a_dtype == AIE_F32 && w_dtype == AIE_F32 && K % 4 == 0 && lda % 4 == 0 && a_bs % 4 == 0 && w_bs % 4 == 0 &&
        !(((size_t)A | (size_t)W) & 15)) {
        if (c_dtype == AIE_F32)
            return gemm_f32_tiled<float>((const float*)A, (const float*)W, (float*)C, a_rows, tile_w, M, N, K, lda, ldc, batch,
                                         a_bs, w_bs, c_bs, stream);
        if (c_dtype == AIE_BF16)
            return gemm_f32_tiled<bf16>((const float*)A, (const float*)W, (bf16*)C, a_rows, tile_w, M, N, K, lda, ldc, batch,
                                        a_bs, w_bs, c_bs, stream);
    }
#define GO(AT, WT) return gemm_f32_go<AT, WT>(A, W, C, c_dtype, a_rows, tile_w, M, N, K, lda, ldc, batch, a_bs, w_bs, c_bs, stream)
    if (a_dtype == AIE_F32 && w_dtype == AIE_F32) GO(float, float);
    if (a_dtype == AIE_F32 && w_dtype == AIE_BF16) GO(float, bf16);
    if (a_dtype == AIE_BF16 && w_dtype == AIE_F32) GO(bf16, float);
    if (a_dtype == AIE_BF16 && w_dtype == AIE_BF16) GO(bf16, bf16);
#undef GO
    return AIE_BAD_ARG;
}

// a_rows (optional): row m of the product reads A[a_rows[m]] (the LM head runs
// only on the rows whose logits are wanted).
extern "C" int aie_gemm_f32(const float* A, const void* W, int w_dtype, float* C, const int* a_rows,
                            int M, int N, int K, int ldc, cudaStream_t stream) {
    return aie_gemm_f32_ex(A, AIE_F32, W, w_dtype, C, AIE_F32, a_rows, nullptr, M, N, K, K, ldc, 1, 0, 0, 0, stream);
}
