// True float32 matrix product on the CUDA cores (FMA; no tensor cores, no TF32):
//   C[M, N] = A[M, K] . W[N, K]^T        (weights as stored by HF: [out, in])
// It is the 32-bit path of every projection and of the LM head.  Each output
// element is one thread's running sum over k = 0 .. K-1 in that order, so a
// row's result does not depend on M: the same token gives the same bits
// whatever else is in the batch.
// The reference multiplies x[B,S,in] by a weight kept as [in,out]
// (crates/ai-engine-runtime/src/arch/linear.rs:106-123); the product is the same.
#include "common.cuh"
#include <type_traits>

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
// The same product for float32 operands whose rows start on 16 bytes: blocks of 64 x 64 or 64 x 128 outputs, a thread TM x 4 of them in
// pairs of rows, so that one packed instruction (fma.rn.f32x2, each half rounded as fmaf) does two multiply-adds: registers
// alone it reaches 62 TFLOP/s here, fmaf 51.  Each output is still one thread's sum over k in order: bits do not depend on
// the tile.  The pairs want the rows next to one another, so tiles of 16 k go through registers into shared memory with k
// outermost, four buffers, two tiles between barriers; a row of k group g lies at row ^ 8 g, which keeps the transposing
// stores off one another's banks.
// Bound by what shared memory hands to registers (512 bytes of a warp in four cycles): 8 x 4 outputs a thread want 12 floats
// for 16 packed instructions, 16 x 4 want 20 for 32 (58 TFLOP/s on large grids; 8 x 8 is 2 % behind, 16 x 8 spills).  The wide
// form has half as many blocks, so which is faster is a matter of rounds (gemm_f32_aligned).
// us, before (64 x 64 tiles of fmaf, k innermost) -> now, weights from memory: 513 tokens 16,384 x 2,048 913 -> 656,
// 2,048 x 8,192 491 -> 433, 3,072 x 2,048 179 -> 159, 2,048 x 2,048 128 -> 110; 2,048 tokens 16,384 x 2,048 3,170 -> 2,453;
// one token 16,384 x 2,048 120 -> 72, 2,048 x 2,048 72 -> 64.
// AHEAD: with one block an SM a tile's latency shows, so its lines are asked into L2 eight tiles early: one token
// 84 -> 64, 200 tokens 2,048 x 8,192 320 -> 280; with more blocks it costs 3 %.
#define GP_M 64
#define GP_K 16
#define GP_THREADS 128

__device__ __forceinline__ unsigned long long gp_pair(float x, float y) {
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ void gp_fma2(unsigned long long& acc, unsigned long long a, unsigned long long b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(acc) : "l"(a), "l"(b));
}

template <int TM, bool AHEAD, typename OT>
__global__ void __launch_bounds__(GP_THREADS, TM == 16 ? 3 : 4)
gemm_f32_pairs_kernel(const float* __restrict__ A, const float* __restrict__ W, OT* __restrict__ C,
                      const int* __restrict__ a_rows, const int* __restrict__ tile_w, int M, int N, int K, int lda, int ldc,
                      long long a_bs, long long w_bs, long long c_bs) {
    // warps lie GP_M / (4 TM) x the rest over the block, a warp's lanes 4 x 8
    constexpr int TN = 4, WM = GP_M / (4 * TM), BN_ = 4 / WM * 8 * TN, PA = GP_M / 32, PW = BN_ / 32, LINES = (GP_M + BN_ + GP_THREADS - 1) / GP_THREADS;
    extern __shared__ __align__(16) float gp_sm[];
    float(*as)[GP_K][GP_M] = reinterpret_cast<float(*)[GP_K][GP_M]>(gp_sm);                       // four buffers each
    float(*ws)[GP_K][BN_] = reinterpret_cast<float(*)[GP_K][BN_]>(gp_sm + 4 * GP_K * GP_M);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, wm = warp % WM, wn = warp / WM;
    const int m0 = blockIdx.y * GP_M, n0 = blockIdx.x * BN_;
    A += (long long)blockIdx.z * a_bs;
    C += (long long)blockIdx.z * c_bs;
    if (tile_w) {
        const int e = tile_w[blockIdx.y];
        if (e < 0) return;
        W += (long long)e * w_bs;
    } else {
        W += (long long)blockIdx.z * w_bs;
    }
    // a thread's pieces of a tile: 16 bytes at column k4 of every 32nd row, the rows of A, then those of W
    const int row0 = tid >> 2, k4 = tid & 3;
    const float* asrc[PA];                          // null: a row of zeros
#pragma unroll
    for (int i = 0; i < PA; ++i) {
        const int m = m0 + row0 + i * 32, r = m < M ? (a_rows ? a_rows[m] : m) : -1;
        asrc[i] = r >= 0 ? A + (size_t)r * lda + k4 * 4 : nullptr;
    }
    const float* wsrc = W + (size_t)(n0 + row0) * K + k4 * 4;
    const int wrows = N - n0 - row0;                // rows 32 i below this are there
    const int blocks = (K + GP_K - 1) / GP_K;
    const float* line[AHEAD ? LINES : 1];           // rows whose lines this thread asks for
    if (AHEAD) {
#pragma unroll
        for (int i = 0; i < LINES; ++i) {
            const int row = tid + i * GP_THREADS, m = m0 + row, n = n0 + row - GP_M;
            line[i] = nullptr;
            if (row < GP_M) {
                const int r = m < M ? (a_rows ? a_rows[m] : m) : -1;
                if (r >= 0) line[i] = A + (size_t)r * lda;
            } else if (row < GP_M + BN_ && n < N) {
                line[i] = W + (size_t)n * K;
            }
        }
    }
    float4 next[PA + PW];
    auto fetch = [&](int kb) {
        const bool in = kb * GP_K + k4 * 4 < K;
#pragma unroll
        for (int i = 0; i < PA; ++i)
            next[i] = in && asrc[i] ? __ldg(reinterpret_cast<const float4*>(asrc[i] + (size_t)kb * GP_K)) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
        for (int i = 0; i < PW; ++i)
            next[PA + i] = in && i * 32 < wrows ? __ldg(reinterpret_cast<const float4*>(wsrc + (size_t)i * 32 * K + (size_t)kb * GP_K))
                                                : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    auto put = [&](int kb) {
        const int s = kb & 3;
#pragma unroll
        for (int i = 0; i < PA + PW; ++i) {
            const int row = (row0 + (i < PA ? i : i - PA) * 32) ^ (8 * k4);
            float* at = i < PA ? &as[s][4 * k4][row] : &ws[s][4 * k4][row];
            const int ld = i < PA ? GP_M : BN_;
            at[0] = next[i].x;
            at[ld] = next[i].y;
            at[2 * ld] = next[i].z;
            at[3 * ld] = next[i].w;
        }
    };
    // a warp's 4 TM rows x 8 TN columns: a lane's rows lm + 16 i + (0 .. 3), its columns ln + (0 .. 3)
    const int lm = wm * 4 * TM + (lane >> 3) * 4, ln = wn * 8 * TN + (lane & 7) * 4;
    unsigned long long acc[TM / 2][TN];             // rows 2 i and 2 i + 1 of the lane's
#pragma unroll
    for (int i = 0; i < TM / 2; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0ull;
    const bool works = m0 + wm * 4 * TM < M;        // a warp whose rows all lie behind M only helps loading
    auto multiply = [&](int kb, auto gc) {
        constexpr int G = decltype(gc)::value;
        const int s = kb & 3;
#pragma unroll
        for (int k = 0; k < GP_K; ++k) {
            const int x = 8 * (k >> 2);
            ulonglong2 a[G];
#pragma unroll
            for (int i = 0; i < G; ++i) a[i] = *reinterpret_cast<const ulonglong2*>(&as[s][k][(lm + 16 * i) ^ x]);
            const float4 w = *reinterpret_cast<const float4*>(&ws[s][k][ln ^ x]);
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                const float wj = j == 0 ? w.x : j == 1 ? w.y : j == 2 ? w.z : w.w;
                const unsigned long long ww = gp_pair(wj, wj);
#pragma unroll
                for (int i = 0; i < G; ++i) {
                    gp_fma2(acc[2 * i][j], a[i].x, ww);
                    gp_fma2(acc[2 * i + 1][j], a[i].y, ww);
                }
            }
        }
    };
    auto walk = [&](auto gc) {
        fetch(0);
        put(0);
        fetch(1);
        put(1);
        __syncthreads();
#pragma unroll 1
        for (int kb = 0; kb < blocks; kb += 2) {    // behind the last block all are zeros
            const bool more = kb + 2 < blocks;
            if (AHEAD && (kb + 8) * GP_K < K) {
#pragma unroll
                for (int i = 0; i < LINES; ++i)
                    if (line[i]) asm volatile("prefetch.global.L2 [%0];" ::"l"(line[i] + (kb + 8) * GP_K));
            }
            if (more) fetch(kb + 2);
            if (works) multiply(kb, gc);
            if (more) {
                put(kb + 2);
                fetch(kb + 3);
            }
            if (works && kb + 1 < blocks) multiply(kb + 1, gc);
            if (more) put(kb + 3);
            __syncthreads();
        }
    };
    // the wide form's warps have all the block's rows, and the same ones: 16 or 32 of them where there are no more
    if (TM == 16 && m0 + 16 >= M) walk(std::integral_constant<int, 1>());
    else if (TM == 16 && m0 + 32 >= M) walk(std::integral_constant<int, 2>());
    else walk(std::integral_constant<int, TM / 4>());
    const bool wide = sizeof(OT) == 4 && ldc % 4 == 0 && (((size_t)C) & 15) == 0;
    const int n = n0 + ln;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + lm + (i >> 2) * 16 + (i & 3);
        if (m >= M) continue;
        float o[TN];
#pragma unroll
        for (int j = 0; j < TN; ++j) o[j] = __uint_as_float((i & 1) ? (unsigned)(acc[i >> 1][j] >> 32) : (unsigned)acc[i >> 1][j]);
        OT* to = C + (size_t)m * ldc + n;
        if (wide && n + TN <= N) {
            *reinterpret_cast<float4*>(to) = make_float4(o[0], o[1], o[2], o[3]);
        } else {
#pragma unroll
            for (int j = 0; j < TN; ++j)
                if (n + j < N) to[j] = from_f32<OT>(o[j]);
        }
    }
}

template <int TM, bool AHEAD, typename OT>
static int gemm_f32_pairs(const float* A, const float* W, OT* C, const int* a_rows, const int* tile_w, int M, int N, int K,
                          int lda, int ldc, int batch, long long a_bs, long long w_bs, long long c_bs, cudaStream_t stream) {
    constexpr int BN_ = 8 * TM, smem = 4 * GP_K * (GP_M + BN_) * 4;
    dim3 grid((N + BN_ - 1) / BN_, (M + GP_M - 1) / GP_M, batch);
    if (grid.y > 65535 || batch > 65535) return AIE_UNSUPPORTED;
    cudaError_t e = cudaFuncSetAttribute(gemm_f32_pairs_kernel<TM, AHEAD, OT>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (e != cudaSuccess) return (int)e;
    gemm_f32_pairs_kernel<TM, AHEAD, OT><<<grid, GP_THREADS, smem, stream>>>(A, W, C, a_rows, tile_w, M, N, K, lda, ldc, a_bs, w_bs, c_bs);
    AIE_LAUNCH_CHECK();
}

// Which form: rounds of blocks over the SMs, a last tile of rows counted by what it takes (in tenths, measured at 1, 33 and 64
// rows) and a tenth of a round let off.  At 2,048 of K a block an SM takes 50 us beside others in the narrow form and 86 in
// the wide one, and 10 and 24 more the first time.  Measured at 66 sizes (1 .. 2,048 rows, six weights) the rule's choice is
// the fastest of the three or within 4 % of it, 7 % at 257 rows of 2,048 columns.
enum { GP_NARROW = 0, GP_AHEAD = 1, GP_WIDE = 2 };      // 64 columns a block, the same with lines asked for early, 128 columns
static int gemm_f32_form(int M, int N, int batch, long long sms) {
    const int rest = M % GP_M;
    const auto rounds = [&](int columns, int last) {
        const long long tenths = (long long)batch * ((N + columns - 1) / columns) * (10 * (M / GP_M) + last);
        return (tenths + 9 * sms - 1) / (10 * sms) + ((tenths + 9 * sms - 1) < 10 * sms);
    };
    const long long narrow = rounds(64, rest == 0 ? 0 : rest <= 32 ? 6 : 10);
    const long long wide = rounds(128, rest == 0 ? 0 : rest <= 16 ? 4 : rest <= 32 ? 6 : 10);
    return 7 * wide + 2 < 4 * narrow + 1 ? GP_WIDE : narrow == 1 ? GP_AHEAD : GP_NARROW;
}
extern "C" int aie_gemm_f32_form(int M, int N, int batch, int sms) { return gemm_f32_form(M, N, batch, sms); }      // for tests

template <typename OT>
static int gemm_f32_aligned(const float* A, const float* W, OT* C, const int* a_rows, const int* tile_w, int M, int N, int K,
                            int lda, int ldc, int batch, long long a_bs, long long w_bs, long long c_bs, cudaStream_t st) {
#define GO(TM, AHEAD) return gemm_f32_pairs<TM, AHEAD, OT>(A, W, C, a_rows, tile_w, M, N, K, lda, ldc, batch, a_bs, w_bs, c_bs, st)
    switch (gemm_f32_form(M, N, batch, aie_sm_count())) {
        case GP_WIDE: GO(16, false);
        case GP_AHEAD: GO(8, true);
        default: GO(8, false);
    }
#undef GO
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
            return gemm_f32_aligned<float>((const float*)A, (const float*)W, (float*)C, a_rows, tile_w, M, N, K, lda, ldc, batch,
                                           a_bs, w_bs, c_bs, stream);
        if (c_dtype == AIE_BF16)
            return gemm_f32_aligned<bf16>((const float*)A, (const float*)W, (bf16*)C, a_rows, tile_w, M, N, K, lda, ldc, batch,
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
