// Plain paged attention: one block per (query token, query head) — all T tokens of
// the step, or the T tokens named by `token_list`; keys are read
// from the layer's pages through the request's block table.  It serves the
// float32 path of the engine and is the reference the fast kernels are checked
// against.  Formula (crates/ai-engine-runtime/src/arch/attention.rs:148-157,
// 177-196, 203-224): query head h reads kv head h / (H/K); s = (q.k) * scale;
// key j is seen by a query at position p iff j <= p (and j > p - window when
// the layer has a window); softmax over keys in float32; out = p.v.
//
// Keys are taken in chunks of 128 that start at multiples of 128 of the
// absolute key position, with a running maximum and sum, so the order of every
// addition depends on the query's position only — not on how the prompt was cut
// into steps or on what else is in the batch.
#include "common.cuh"

#define PLAIN_CHUNK 128

template <typename A, typename C>
__global__ void __launch_bounds__(PLAIN_CHUNK)
paged_attention_plain_kernel(const A* __restrict__ q, const C* __restrict__ k_pages,
                             const C* __restrict__ v_pages, A* __restrict__ out,
                             const int* __restrict__ positions, const int* __restrict__ token_req,
                             const int* __restrict__ block_table, int bt_width, int num_pages,
                             int P, int H, int K, int d, int window, float scale,
                             const int* __restrict__ token_list, unsigned* err) {
    extern __shared__ __align__(16) float sm[];
    float* q_s = sm;                                  // d
    float* p_s = q_s + d;                             // CHUNK
    float* red = p_s + PLAIN_CHUNK;                   // 32
    long long* off_s = (long long*)(red + 32);        // CHUNK  (8-byte aligned: d is a multiple of 2)

    const int t = token_list ? token_list[blockIdx.x] : blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int pos = positions[t];
    const int row = token_req[t];
    const int kvh = h / (H / K);
    for (int e = tid; e < d; e += blockDim.x) q_s[e] = to_f32<A>(q[((size_t)t * H + h) * d + e]);
    __syncthreads();

    int lo = 0;
    if (window > 0 && pos - window + 1 > 0) lo = pos - window + 1;
    float m = -INFINITY, l = 0.f;
    float acc0 = 0.f, acc1 = 0.f;  // output elements tid and tid + 128 (d <= 256)

    for (int c0 = (lo / PLAIN_CHUNK) * PLAIN_CHUNK; c0 <= pos; c0 += PLAIN_CHUNK) {
        const int kp = c0 + tid;
        const bool valid = kp >= lo && kp <= pos;
        float s = -INFINITY;
        long long off = -1;
        if (valid) {
            const int pidx = kp / P;
            const int page = pidx < bt_width ? block_table[(size_t)row * bt_width + pidx] : -1;
            if (page < 0 || page >= num_pages) {
                atomicOr(err, AIE_DEV_PAGE_OOB);
            } else {
                off = (((long long)page * K + kvh) * P + (kp % P)) * d;
                const C* kr = k_pages + off;
                float dot = 0.f;
                for (int e = 0; e < d; ++e) dot += q_s[e] * to_f32<C>(kr[e]);
                s = dot * scale;
            }
        }
        off_s[tid] = off;
        const float cmax = block_max(s, red);
        const float m_new = fmaxf(m, cmax);
        // every chunk visited holds at least one visible key unless a page was bad
        const float p = (off >= 0) ? expf(s - m_new) : 0.f;
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        p_s[tid] = p;
        const float csum = block_sum(p, red);   // has __syncthreads inside: p_s, off_s visible
        l = l * corr + csum;
        m = m_new;
        acc0 *= corr;
        acc1 *= corr;
        const int n = min(PLAIN_CHUNK, pos - c0 + 1);
        for (int j = 0; j < n; ++j) {
            const long long o = off_s[j];
            if (o < 0) continue;
            const float pj = p_s[j];
            if (tid < d) acc0 += pj * to_f32<C>(v_pages[o + tid]);
            if (tid + PLAIN_CHUNK < d) acc1 += pj * to_f32<C>(v_pages[o + tid + PLAIN_CHUNK]);
        }
        __syncthreads();
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    A* o = out + ((size_t)t * H + h) * d;
    if (tid < d) o[tid] = from_f32<A>(acc0 * inv);
    if (tid + PLAIN_CHUNK < d) o[tid + PLAIN_CHUNK] = from_f32<A>(acc1 * inv);
}

extern "C" int aie_paged_attention_plain(const void* q, const void* k_pages, const void* v_pages,
                                         void* out, int dtype, const int* positions,
                                         const int* token_req, const int* block_table, int bt_width,
                                         int num_pages, int P, int T, int H, int K, int d, int window,
                                         float scale, const int* token_list, unsigned* err,
                                         cudaStream_t stream) {
    if (T <= 0) return 0;
    if (d <= 0 || d > 2 * PLAIN_CHUNK || (d % 2) || K <= 0 || H % K) return AIE_UNSUPPORTED;
    const size_t smem = (size_t)(d + PLAIN_CHUNK + 32) * sizeof(float) + PLAIN_CHUNK * sizeof(long long);
    if (H > 65535) return AIE_UNSUPPORTED;
    dim3 grid(T, H);
    if (dtype == AIE_F32)
        paged_attention_plain_kernel<float, float><<<grid, PLAIN_CHUNK, smem, stream>>>(
            (const float*)q, (const float*)k_pages, (const float*)v_pages, (float*)out, positions,
            token_req, block_table, bt_width, num_pages, P, H, K, d, window, scale, token_list, err);
    else if (dtype == AIE_BF16)
        paged_attention_plain_kernel<bf16, bf16><<<grid, PLAIN_CHUNK, smem, stream>>>(
            (const bf16*)q, (const bf16*)k_pages, (const bf16*)v_pages, (bf16*)out, positions,
            token_req, block_table, bt_width, num_pages, P, H, K, d, window, scale, token_list, err);
    else
        return AIE_BAD_ARG;
    AIE_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The same for portions of prompts in float32, 64 query tokens of one request and one head a block: keys and values of a
// chunk are read once for all of them, scores and outputs are tiles of FMAs.  A block's additions are those of the kernel
// above, in its order (the dot product over e, the butterfly sum of a chunk's 128 weights, the values over j), and keys that a
// query does not see take no part in them (their values may be infinities), so a token's bits do not depend on which of
// the two computes it.  Bound by the FMA units and, for few heads and tokens, by
// the longest block's chain of chunks.
// A warp owns 16 query rows; lanes lie 4 x 8: rows lm + 4 i, keys ln + 8 j, output columns 4 (ln + 8 x) .. + 3.
#define PT_Q 64
#define PT_THREADS 128

template <int ND>      // pieces of 32 output columns: d <= 32 ND
__global__ void __launch_bounds__(PT_THREADS)
paged_attention_f32_tiles_kernel(const float* __restrict__ q, const float* __restrict__ k_pages, const float* __restrict__ v_pages,
                                 float* __restrict__ out, const int* __restrict__ tiles, int per_tile, const int* __restrict__ q_start,
                                 const int* __restrict__ q_len, const int* __restrict__ ctx_len, const int* __restrict__ block_table,
                                 int bt_width, int num_pages, int P, int H, int K, int d, int window, float scale, unsigned* err) {
    extern __shared__ __align__(16) float pt_sm[];
    const int ld = d + 4, ldp = PLAIN_CHUNK + 4;                 // padded rows: lanes' rows fall on different banks
    float* q_s = pt_sm;                                          // [64][ld]
    float* v_s = q_s + PT_Q * ld;                                // [128][d]
    float* k_s = v_s + PLAIN_CHUNK * d;                          // [128][ld], then the weights [64][ldp]
    float* p_s = k_s;
    int* ok_s = reinterpret_cast<int*>(k_s + max(PLAIN_CHUNK * ld, PT_Q * ldp));      // [128]

    const int row = tiles[2 * (blockIdx.x / per_tile)], off = tiles[2 * (blockIdx.x / per_tile) + 1] + PT_Q * (blockIdx.x % per_tile);
    const int n = min(PT_Q, q_len[row] - off), h = blockIdx.y, kvh = h / (H / K);
    if (n <= 0) return;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, lm = lane >> 3, ln = lane & 7;
    const int pos0 = ctx_len[row] + off, last = pos0 + n - 1, t0 = q_start[row] + off, d4 = d / 4;
    const int lo0 = (window > 0 && pos0 - window + 1 > 0) ? pos0 - window + 1 : 0;
    auto copy = [](float* dst, const float* src, bool ok) {
        const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(src), "r"(ok ? 16 : 0) : "memory");
    };
    for (int i = tid; i < PT_Q * d4; i += PT_THREADS) {
        const int r = i / d4, c = (i % d4) * 4;
        copy(q_s + r * ld + c, r < n ? q + ((size_t)(t0 + r) * H + h) * d + c : q, r < n);
    }
    const bool works = warp * 16 < n;
    float m[4], l[4];
    float4 acc[4][ND];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int x = 0; x < ND; ++x) acc[i][x] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int c0 = (lo0 / PLAIN_CHUNK) * PLAIN_CHUNK; c0 <= last; c0 += PLAIN_CHUNK) {
        __syncthreads();                                         // the previous chunk is done with
        const int kp = c0 + tid;
        int page = -1;
        if (kp >= lo0 && kp <= last) {
            const int pidx = kp / P;
            page = pidx < bt_width ? block_table[(size_t)row * bt_width + pidx] : -1;
            if (page < 0 || page >= num_pages) {
                atomicOr(err, AIE_DEV_PAGE_OOB);
                page = -1;
            }
        }
        ok_s[tid] = page < 0 ? -1 : page * P + kp % P;           // page and place of the key
        __syncthreads();
        for (int i = tid; i < PLAIN_CHUNK * d4; i += PT_THREADS) {
            const int j = i / d4, c = (i % d4) * 4, at = ok_s[j], pg = at / P;
            copy(k_s + j * ld + c, at >= 0 ? k_pages + (((size_t)pg * K + kvh) * P + (at - pg * P)) * d + c : k_pages, at >= 0);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        for (int i = tid; i < PLAIN_CHUNK * d4; i += PT_THREADS) {
            const int j = i / d4, c = (i % d4) * 4, at = ok_s[j], pg = at / P;
            copy(v_s + j * d + c, at >= 0 ? v_pages + (((size_t)pg * K + kvh) * P + (at - pg * P)) * d + c : v_pages, at >= 0);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        __syncthreads();
        float s[4][16];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 16; ++j) s[i][j] = 0.f;
        if (works) {
            const float* qr = q_s + (warp * 16 + lm) * ld;
            const float* kr = k_s + ln * ld;
#pragma unroll 1
            for (int e = 0; e < d; e += 2) {
                float2 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float2*>(qr + 4 * i * ld + e);
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const float2 b = *reinterpret_cast<const float2*>(kr + 8 * j * ld + e);
#pragma unroll
                    for (int i = 0; i < 4; ++i) s[i][j] = fmaf(a[i].y, b.y, fmaf(a[i].x, b.x, s[i][j]));
                }
            }
            unsigned seen = 0;                                   // bit j: the page of key ln + 8 j is there
#pragma unroll
            for (int j = 0; j < 16; ++j) seen |= (ok_s[ln + 8 * j] >= 0 ? 1u : 0u) << j;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int pos = pos0 + warp * 16 + lm + 4 * i;
                const int lo = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
                float mx = -INFINITY;
                unsigned sees = 0;
#pragma unroll
                for (int j = 0; j < 16; ++j) {
                    const int key = c0 + ln + 8 * j;
                    const bool see = ((seen >> j) & 1) && key >= lo && key <= pos;
                    sees |= (see ? 1u : 0u) << j;
                    s[i][j] = see ? s[i][j] * scale : -INFINITY;
                    mx = fmaxf(mx, s[i][j]);
                }
#pragma unroll
                for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_new = fmaxf(m[i], mx);
                float w[4];
#pragma unroll
                for (int g = 0; g < 4; ++g) {                    // 32 keys: the butterfly 16, 8, then 4, 2, 1 over the lanes
#pragma unroll
                    for (int x = 0; x < 4; ++x)
                        s[i][4 * g + x] = (sees >> (4 * g + x)) & 1 ? expf(s[i][4 * g + x] - m_new) : 0.f;
                    w[g] = (s[i][4 * g] + s[i][4 * g + 2]) + (s[i][4 * g + 1] + s[i][4 * g + 3]);
#pragma unroll
                    for (int o = 4; o > 0; o >>= 1) w[g] += __shfl_xor_sync(0xffffffffu, w[g], o);
                }
                // a chunk that the query has no key in leaves its sums alone
                const bool here = c0 <= pos && c0 + PLAIN_CHUNK > lo;
                const float corr = !here ? 1.f : (m[i] == -INFINITY) ? 0.f : expf(m[i] - m_new);
                if (here) l[i] = l[i] * corr + ((w[0] + w[2]) + (w[1] + w[3]));
                m[i] = m_new;
#pragma unroll
                for (int x = 0; x < ND; ++x) {
                    acc[i][x].x *= corr;
                    acc[i][x].y *= corr;
                    acc[i][x].z *= corr;
                    acc[i][x].w *= corr;
                }
            }
        }
        __syncthreads();                                         // all warps have read the keys: the weights take their place
        if (works) {
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 16; ++j) p_s[(warp * 16 + lm + 4 * i) * ldp + ln + 8 * j] = s[i][j];
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
        if (works) {
            const float* pr = p_s + (warp * 16 + lm) * ldp;
            const int nk = min(PLAIN_CHUNK, last - c0 + 1);
            // the warp's rows from .. to (keys of the chunk) that all its queries see: outside of it each query is asked
            const int first = pos0 + warp * 16, lo_last = window > 0 ? max(min(first + 15, last) - window + 1, 0) : 0;
            const int from = lo_last - c0, to = first - c0;
#pragma unroll 1
            for (int j = 0; j < nk; j += 2) {                    // a key behind the last has weight and value 0
                float2 a[4];
#pragma unroll
                for (int i = 0; i < 4; ++i) a[i] = *reinterpret_cast<const float2*>(pr + 4 * i * ldp + j);
                if (j < from || j + 1 > to) {
#pragma unroll 1
                    for (int y = 0; y < 2; ++y) {
                        const int key = c0 + j + y;
                        bool sees[4];
#pragma unroll
                        for (int i = 0; i < 4; ++i) {
                            const int pos = first + lm + 4 * i;
                            sees[i] = key <= pos && (window <= 0 || key > pos - window);
                        }
#pragma unroll
                        for (int x = 0; x < ND; ++x) {
                            const int c = 4 * (ln + 8 * x);
                            if (c >= d) continue;
                            const float4 b = *reinterpret_cast<const float4*>(v_s + (j + y) * d + c);
#pragma unroll
                            for (int i = 0; i < 4; ++i)
                                if (sees[i]) {
                                    const float w = y ? a[i].y : a[i].x;
                                    acc[i][x].x = fmaf(w, b.x, acc[i][x].x);
                                    acc[i][x].y = fmaf(w, b.y, acc[i][x].y);
                                    acc[i][x].z = fmaf(w, b.z, acc[i][x].z);
                                    acc[i][x].w = fmaf(w, b.w, acc[i][x].w);
                                }
                        }
                    }
                    continue;
                }
#pragma unroll
                for (int x = 0; x < ND; ++x) {
                    const int c = 4 * (ln + 8 * x);
                    if (c >= d) continue;
                    const float4 b0 = *reinterpret_cast<const float4*>(v_s + j * d + c);
                    const float4 b1 = *reinterpret_cast<const float4*>(v_s + (j + 1) * d + c);
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        acc[i][x].x = fmaf(a[i].y, b1.x, fmaf(a[i].x, b0.x, acc[i][x].x));
                        acc[i][x].y = fmaf(a[i].y, b1.y, fmaf(a[i].x, b0.y, acc[i][x].y));
                        acc[i][x].z = fmaf(a[i].y, b1.z, fmaf(a[i].x, b0.z, acc[i][x].z));
                        acc[i][x].w = fmaf(a[i].y, b1.w, fmaf(a[i].x, b0.w, acc[i][x].w));
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = warp * 16 + lm + 4 * i;
        if (r >= n) continue;
        const float inv = l[i] > 0.f ? 1.0f / l[i] : 0.f;
        float* o = out + ((size_t)(t0 + r) * H + h) * d;
#pragma unroll
        for (int x = 0; x < ND; ++x) {
            const int c = 4 * (ln + 8 * x);
            if (c < d) *reinterpret_cast<float4*>(o + c) = make_float4(acc[i][x].x * inv, acc[i][x].y * inv, acc[i][x].z * inv, acc[i][x].w * inv);
        }
    }
}

// q, out [T, H, d], pages [num_pages, K, P, d] float32, all starting on 16 bytes; tiles [n_tiles, 2] = (request row, offset
// of `tile` tokens among those it brings), tile a multiple of 64.  d <= 128 in steps of 4 (else AIE_UNSUPPORTED: the
// caller takes the kernel above).  Tokens that no tile names are left.
extern "C" int aie_paged_attention_f32_tiles(const float* q, const float* k_pages, const float* v_pages, float* out, const int* tiles,
                                             int n_tiles, int tile, const int* q_start, const int* q_len, const int* ctx_len,
                                             const int* block_table, int bt_width, int num_pages, int P, int H, int K, int d,
                                             int window, float scale, unsigned* err, cudaStream_t st) {
    if (n_tiles <= 0) return 0;
    if (d <= 0 || d > 128 || d % 4 || K <= 0 || H % K || H > 65535 || tile <= 0 || tile % PT_Q || P <= 0 ||
        (long long)num_pages * P > 0x7fffffffLL || (((size_t)q | (size_t)k_pages | (size_t)v_pages | (size_t)out) & 15))
        return AIE_UNSUPPORTED;
    const int ld = d + 4, ldp = PLAIN_CHUNK + 4;
    const size_t keys = PLAIN_CHUNK * ld > PT_Q * ldp ? (size_t)PLAIN_CHUNK * ld : (size_t)PT_Q * ldp;
    const size_t smem = ((size_t)PT_Q * ld + (size_t)PLAIN_CHUNK * d + keys) * sizeof(float) + PLAIN_CHUNK * sizeof(int);
    const dim3 grid((unsigned)n_tiles * (tile / PT_Q), H);
#define GO(ND)                                                                                                              \
    {                                                                                                                       \
        cudaError_t e = cudaFuncSetAttribute(paged_attention_f32_tiles_kernel<ND>, cudaFuncAttributeMaxDynamicSharedMemorySize, \
                                             (int)smem);                                                                    \
        if (e != cudaSuccess) return (int)e;                                                                                \
        paged_attention_f32_tiles_kernel<ND><<<grid, PT_THREADS, smem, st>>>(q, k_pages, v_pages, out, tiles, tile / PT_Q,   \
            q_start, q_len, ctx_len, block_table, bt_width, num_pages, P, H, K, d, window, scale, err);                     \
    }
    switch ((d + 31) / 32) {
        case 1: GO(1) break;
        case 2: GO(2) break;
        case 3: GO(3) break;
        default: GO(4)
    }
#undef GO
    AIE_LAUNCH_CHECK();
}
