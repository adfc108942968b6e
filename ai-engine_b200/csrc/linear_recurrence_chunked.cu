// Linear attention with a decaying matrix state over portions of prompts, parallel over chunks of 64 tokens, in float32:
//     S_t = diag(a_t) S_(t-1) + k_t v_t^T,    o_t = q_scale S_t^T q_t            (S: [d, dv] per request and head)
// Token by token (linear_recurrence.cu) this is a chain of dependent updates: 2,048 tokens x 16 heads of 128 x 128 took
// 942 us, bound by the latency of that chain with 256 blocks in flight.  Three kernels take its place:
//   chunk:  L_c = sum_j (k_j prod_{s > j} a_s) v_j^T and the chunk's decay G_c, every (chunk, head) on its own
//   scan:   S_c+1 = G_c S_c + L_c over a request's chunks, every element on its own; L_c is replaced by S_c
//   out:    o_i = (q_i prod_{s <= i} a_s)^T S_c + sum_{j <= i} A_ij v_j,  A_ij = sum_ch q_i k_j prod_{j < s <= i} a_s
// Decays enter as products only (no logarithms, no quotients): of the decays behind a key up to the end of its part of
// the chunk and of those up to a query from the start of its part, parts being the halves of 64 and 32 tokens; blocks of
// 16 tokens on the diagonal walk their pairs.  Every factor is at most one, nothing overflows, and a far pair's
// product underflows to the zero it stands for.  All sums and products are float32 on the FMA units, as they were: one
// bfloat16 or TF32 term would lose bits of keys, queries and the state, and three terms cost what this does.
// What bounds it: the products' multiply-adds (2.7 M per chunk and head of 128 x 128); those 2,048 tokens: 41 + 9 + 86 us.
#include "chunk_find.cuh"

#define LC_T 64             // tokens of a chunk
#define LC_THREADS 256

struct LcArgs {
    const float *q, *k, *v, *decay_tok, *decay_head, *fg_lower, *fg_bias;
    float *state, *out, *L, *G;
    const int *q_start, *q_len, *slots;
    unsigned* err;
    int ld, ld_decay, H, all_heads, R, d, dv, max_slots, min_len;      // H: the heads of this launch, neighbours of all_heads
    float q_scale, k_scale;
};

__device__ __forceinline__ float4 f4(float x) { return make_float4(x, x, x, x); }
__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ void fma4(float4& acc, float x, const float4& v) {
    acc = make_float4(fmaf(x, v.x, acc.x), fmaf(x, v.y, acc.y), fmaf(x, v.z, acc.z), fmaf(x, v.w, acc.w));
}
__device__ __forceinline__ float lane4(const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : (i == 2 ? v.z : v.w)); }

__device__ __forceinline__ void lc_fetch(float* dst, const float* src, bool ok) {      // 16 bytes; zeros when not ok
    const unsigned to = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"(to), "l"(src), "r"(ok ? 16 : 0) : "memory");
}
__device__ __forceinline__ void lc_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N> __device__ __forceinline__ void lc_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }
__device__ __forceinline__ float lc_gate(float z, float lo) { return lo + (1.0f - lo) * (1.0f / (1.0f + expf(-z))); }
__device__ __forceinline__ float lc_silu(float x) { return x / (1.0f + expf(-x)); }

// Rows of a chunk in shared memory, [64][D]; channels behind d and tokens behind the portion's end change nothing (keys,
// queries and values 0, decays 1).  All copies of a thread are on their way at once (through registers they came a few
// at a time and this took half the kernel); what the keyless form or a scale makes of them, a thread makes of its own
// pieces.  SWZ: a key's pieces of four channels lie at piece ^ (token & 7).  qs null: keys and decays only.
template <int D, bool SWZ>
__device__ __forceinline__ void lc_load_rows(const LcArgs& p, float* qs, float* ks, float* as, size_t a0, int nt, int h) {
    constexpr int N = LC_T * D / 4 / LC_THREADS;
#pragma unroll
    for (int it = 0; it < N; ++it) {
        const int i = threadIdx.x + it * LC_THREADS, t = i / (D / 4), c4 = i % (D / 4), c = c4 * 4;
        const bool ok = t < nt && c < p.d;
        const size_t at = ok ? (a0 + t) * p.ld + (size_t)h * p.d + c : 0;
        if (p.decay_tok) lc_fetch(as + i * 4, p.decay_tok + (ok ? (a0 + t) * p.ld_decay + (size_t)h * p.d + c : 0), ok);
        if (p.k) lc_fetch(ks + (t * (D / 4) + (SWZ ? c4 ^ (t & 7) : c4)) * 4, p.k + at, ok);
        if (qs) lc_fetch(qs + i * 4, p.q + at, ok);
    }
    lc_commit();
    lc_wait<0>();
#pragma unroll
    for (int it = 0; it < N; ++it) {
        const int i = threadIdx.x + it * LC_THREADS, t = i / (D / 4), c4 = i % (D / 4), c = c4 * 4;
        const bool ok = t < nt && c < p.d;
        float4* ap = reinterpret_cast<float4*>(as + i * 4);
        float4* kp = reinterpret_cast<float4*>(ks + (t * (D / 4) + (SWZ ? c4 ^ (t & 7) : c4)) * 4);
        if (!ok) {
            *ap = f4(1.f);
            if (!p.k) *kp = f4(0.f);
        } else if (p.fg_lower) {
            const float4 lo = *reinterpret_cast<const float4*>(p.fg_lower + h * p.d + c);
            const float4 b = p.fg_bias ? *reinterpret_cast<const float4*>(p.fg_bias + h * p.d + c) : f4(0.f);
            float4 a = *ap;
            a = make_float4(lc_gate(a.x + b.x, lo.x), lc_gate(a.y + b.y, lo.y), lc_gate(a.z + b.z, lo.z), lc_gate(a.w + b.w, lo.w));
            *ap = a;
            *kp = make_float4(1.0f - a.x, 1.0f - a.y, 1.0f - a.z, 1.0f - a.w);
            if (qs) {
                float4* qp = reinterpret_cast<float4*>(qs + i * 4);
                const float4 q = *qp;
                *qp = make_float4(lc_silu(q.x), lc_silu(q.y), lc_silu(q.z), lc_silu(q.w));
            }
        } else {
            if (!p.decay_tok) *ap = f4(p.decay_head[h]);
            if (p.k_scale != 1.f) *kp = mul4(*kp, f4(p.k_scale));
        }
    }
}
template <int D>
__device__ __forceinline__ void lc_load_values(const LcArgs& p, float* vs, size_t a0, int nt, int h) {
#pragma unroll
    for (int it = 0; it < LC_T * D / 4 / LC_THREADS; ++it) {
        const int i = threadIdx.x + it * LC_THREADS, t = i / (D / 4), c = (i % (D / 4)) * 4;
        const bool ok = t < nt && c < p.dv;
        lc_fetch(vs + i * 4, p.v + (ok ? (a0 + t) * p.ld + (size_t)h * p.dv + c : 0), ok);
    }
    lc_commit();
}

// L_c and G_c of one (chunk, head): K'^T V with K'_j = k_j times the decays behind it.  Two blocks an SM; a thread owns
// D / 16 rows x DV / 16 columns of L (8 x 8 at the largest: 16 x 4 a thread read a third more from shared memory).
template <int D, int DV>
__global__ void __launch_bounds__(LC_THREADS, 2) lc_chunk_kernel(LcArgs p) {
    extern __shared__ __align__(16) float lc_sm[];
    __shared__ int found[2];
    float* ks = lc_sm;                 // [64][D]
    float* as = ks + LC_T * D;         // [64][D]
    float* vs = as + LC_T * D;         // [64][DV]
    const int tid = threadIdx.x, h = blockIdx.y;
    int r, c;
    chunk_find<LC_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(LC_T, p.q_len[r] - c * LC_T);
    const size_t a0 = (size_t)p.q_start[r] + c * LC_T;
    lc_load_values<DV>(p, vs, a0, nt, h);
    lc_load_rows<D, false>(p, nullptr, ks, as, a0, nt, h);
    __syncthreads();
    // keys times the decays behind them: two threads a channel, the first half of the tokens also takes the second's
    if (tid < 2 * D) {
        const int ch = tid % D, half = tid / D;
        float run = 1.f;
        if (half == 0) {
#pragma unroll 8
            for (int j = 32; j < LC_T; ++j) run *= as[j * D + ch];
        }
#pragma unroll 8
        for (int j = 31; j >= 0; --j) {
            const int t = half * 32 + j;
            ks[t * D + ch] *= run;
            run *= as[t * D + ch];
        }
        if (half == 0 && ch < p.d) p.G[((size_t)blockIdx.x * p.H + h) * p.d + ch] = run;
    }
    __syncthreads();
    constexpr int RPT = D / 16, NC = DV / 64;
    const int col = (tid & 15) * 4, row0 = (tid >> 4) * RPT;
    float4 acc[RPT][NC];
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int x = 0; x < NC; ++x) acc[i][x] = f4(0.f);
#pragma unroll 2
    for (int t = 0; t < LC_T; ++t) {
        float4 v[NC];
#pragma unroll
        for (int x = 0; x < NC; ++x) v[x] = *reinterpret_cast<const float4*>(vs + t * DV + x * 64 + col);
#pragma unroll
        for (int i = 0; i < RPT; i += 4) {
            const float4 k4 = *reinterpret_cast<const float4*>(ks + t * D + row0 + i);
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll
                for (int x = 0; x < NC; ++x) fma4(acc[i + e][x], lane4(k4, e), v[x]);
        }
    }
    float* L = p.L + ((size_t)blockIdx.x * p.H + h) * p.d * p.dv;
#pragma unroll
    for (int i = 0; i < RPT; ++i)
#pragma unroll
        for (int x = 0; x < NC; ++x)
            if (row0 + i < p.d && x * 64 + col < p.dv)
                *reinterpret_cast<float4*>(L + (size_t)(row0 + i) * p.dv + x * 64 + col) = acc[i][x];
}

// S_c for every chunk of a request and the state behind the last; bound by the traffic of L (in L2).  A thread owns
// four elements; eight chunks' loads are in flight while the chain of multiply-adds runs.
__global__ void __launch_bounds__(LC_THREADS) lc_scan_kernel(LcArgs p) {
    __shared__ int found[2];
    const int h = blockIdx.y % p.H;
    int r, first;
    portion_find<LC_T>(p.q_len, p.R, p.min_len, blockIdx.y / p.H, found, r, first);
    if (r < 0) return;
    const int n = chunk_count<LC_T>(p.q_len, p.R, p.min_len, r), slot = p.slots[r];
    if (slot < 0 || slot >= p.max_slots) {
        if (threadIdx.x == 0) atomicOr(p.err, AIE_DEV_SLOT_OOB);
        return;
    }
    const int e = (blockIdx.x * LC_THREADS + threadIdx.x) * 4, size = p.d * p.dv;
    if (e >= size) return;
    const int row = e / p.dv;
    float* sp = p.state + ((size_t)slot * p.all_heads + h) * size + e;
    float* L = p.L + ((size_t)first * p.H + h) * size + e;
    const float* G = p.G + ((size_t)first * p.H + h) * p.d + row;
    const size_t ls = (size_t)p.H * size, gs = (size_t)p.H * p.d;
    float4 S = *reinterpret_cast<const float4*>(sp);
    for (int c = 0; c < n; c += 8) {
        float4 l[8];
        float g[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < n) {
                l[i] = *reinterpret_cast<const float4*>(L + (c + i) * ls);
                g[i] = G[(c + i) * gs];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < n) {
                *reinterpret_cast<float4*>(L + (c + i) * ls) = S;
                S = make_float4(fmaf(g[i], S.x, l[i].x), fmaf(g[i], S.y, l[i].y), fmaf(g[i], S.z, l[i].z), fmaf(g[i], S.w, l[i].w));
            }
    }
    *reinterpret_cast<float4*>(sp) = S;
}

// Pairs of one block of 16 tokens on the diagonal: two warps a block (half 0 takes keys 0, 3, 4, 7, ..., half 1 the others:
// as many pairs), a lane owns D / 32 channels.  Eight keys walk the block's queries with the decays between multiplied on;
// a query's eight sums are added over the lanes together.  Loops here and below are kept short on purpose: unrolled, the
// kernel waited for its instructions more than for anything else.
template <int D>
__device__ __forceinline__ void lc_diagonal(const float* qs, const float* ks, const float* as, float* A, int b, int half, int lane) {
    constexpr int V = D / 32;
    float w[8][V];
#pragma unroll 1
    for (int i = 0; i < 16; ++i) {
        const int t = 16 * b + i;
        float qv[V], av[V], s[8];
#pragma unroll
        for (int x = 0; x < V; ++x) {
            qv[x] = qs[t * D + lane * V + x];
            av[x] = as[t * D + lane * V + x];
        }
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            const int j = 2 * m + ((m & 1) ^ half);
            s[m] = 0.f;
            if (i < j) continue;
#pragma unroll
            for (int x = 0; x < V; ++x) {
                if (i == j)
                    w[m][x] = ks[t * D + ((((lane * V) >> 2) ^ (t & 7)) << 2) + ((lane * V) & 3) + x];
                else
                    w[m][x] *= av[x];
                s[m] = fmaf(qv[x], w[m][x], s[m]);
            }
        }
        // eight sums over 32 lanes: three exchanges leave a lane with one of them, two more finish it
#pragma unroll
        for (int n = 4; n >= 1; n >>= 1) {
            const int o = 4 * n;
#pragma unroll
            for (int m = 0; m < n; ++m) {
                const float give = (lane & o) ? s[m] : s[m + n], keep = (lane & o) ? s[m + n] : s[m];
                s[m] = keep + __shfl_xor_sync(0xffffffffu, give, o);
            }
        }
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 2);
        s[0] += __shfl_xor_sync(0xffffffffu, s[0], 1);
        const int m = ((lane >> 4) & 1) * 4 + ((lane >> 3) & 1) * 2 + ((lane >> 2) & 1);
        if ((lane & 3) == 0) A[t * LC_T + 16 * b + 2 * m + ((m & 1) ^ half)] = s[0];
    }
}

// s[4 a + b] = q_(i0 + a) . k_(j0 + b) over every SHARES-th piece of four channels: 8 loads of 16 bytes for 64 multiply-adds (a dot
// product a thread, 2 or 4 of them with the same key, took 3 or 5 for 8 or 16: all three kernels at 300 /
// 1,024 / 2,048 / 4,000 tokens x 16 heads 49.5 / 73.9 / 139.4 / 245.9 -> 48.2 / 71.8 / 137.3 / 243.3 us, the
// middle halves of 40 runs each within 0.2; ragged prompts in two steps 257 -> 253).  at: the share, and which of the
// piece's neighbours comes first: threads that read other rows side by side start on other banks.
template <int D, int SHARES>
__device__ __forceinline__ void lc_pairs(const float* qs, const float* ks, int i0, int j0, int at, float* s) {
#pragma unroll
    for (int m = 0; m < 16; ++m) s[m] = 0.f;
#pragma unroll 1
    for (int c = 0; c < D / 4; c += SHARES) {
        const int c4 = SHARES == 8 ? c + at : c ^ at;
        float4 k4[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) k4[b] = reinterpret_cast<const float4*>(ks)[(j0 + b) * (D / 4) + (c4 ^ ((j0 + b) & 7))];
#pragma unroll
        for (int a = 0; a < 4; ++a) {
            const float4 q4 = *reinterpret_cast<const float4*>(qs + (i0 + a) * D + c4 * 4);
#pragma unroll
            for (int b = 0; b < 4; ++b)
                s[4 * a + b] = fmaf(q4.x, k4[b].x, fmaf(q4.y, k4[b].y, fmaf(q4.z, k4[b].z, fmaf(q4.w, k4[b].w, s[4 * a + b]))));
        }
    }
}
// N sums over LANES neighbouring lanes; a lane is left with N / LANES of them, from the one that is returned on.
template <int N, int LANES>
__device__ __forceinline__ int lc_gather(float* s, int lane) {
    int first = 0;
#pragma unroll
    for (int o = LANES / 2, n = N / 2; o >= 1; o >>= 1, n >>= 1) {
#pragma unroll
        for (int m = 0; m < n; ++m) {
            const float give = (lane & o) ? s[m] : s[m + n], keep = (lane & o) ? s[m + n] : s[m];
            s[m] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
        if (lane & o) first += n;
    }
    return first;
}

template <int D, int DV>
__global__ void __launch_bounds__(LC_THREADS, 2) lc_out_kernel(LcArgs p) {
    extern __shared__ __align__(16) float lc_sm[];
    __shared__ int found[2];
    constexpr int KD = D > DV ? D : DV;
    float* qs = lc_sm;                 // [64][D]
    float* ks = qs + LC_T * D;         // [64][D], a row's pieces of four channels at piece ^ (token & 7); later v [64][DV]
    float* as = ks + LC_T * KD;        // [64][D]; later slices of S, [16][DV] each
    float* A = as + LC_T * D;          // [64][64]
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y;
    int r, c;
    chunk_find<LC_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(LC_T, p.q_len[r] - c * LC_T);
    const size_t a0 = (size_t)p.q_start[r] + c * LC_T;
    lc_load_rows<D, true>(p, qs, ks, as, a0, nt, h);
    __syncthreads();
    lc_diagonal<D>(qs, ks, as, A, warp >> 1, warp & 1, lane);
    __syncthreads();
    // queries times the decays from their block's start, keys times those behind them in their block; the blocks'
    // products go where A is never read: rows 0 .. 31, columns 32 .. 63
#define LC_G(b, ch) A[(((b) * D + (ch)) >> 5) * LC_T + 32 + ((ch) & 31)]
    for (int u = tid; u < 4 * D; u += LC_THREADS) {
        const int b = u / D, ch = u % D;
        float run = 1.f, dec[16];
#pragma unroll
        for (int i = 0; i < 16; ++i) {
            const int t = 16 * b + i;
            dec[i] = as[t * D + ch];
            run *= dec[i];
            qs[t * D + ch] *= run;
        }
        LC_G(b, ch) = run;
        run = 1.f;
#pragma unroll
        for (int i = 15; i >= 0; --i) {
            const int t = 16 * b + i;
            ks[t * D + (((ch >> 2) ^ (t & 7)) << 2) + (ch & 3)] *= run;
            run *= dec[i];
        }
    }
    __syncthreads();
    // pairs of neighbouring blocks: rows 16 .. 31 with columns 0 .. 15, rows 48 .. 63 with columns 32 .. 47.  A thread has 4 x 4 of them
    // over one of eight shares of the channels
    {
        const int id = 4 * warp + (lane >> 3), base = (id >> 4) * 32, j0 = base + 4 * (id & 3), i0 = base + 16 + (id & 12);
        float s[16];
        lc_pairs<D, 8>(qs, ks, i0, j0, lane & 7, s);
        const int m = lc_gather<16, 8>(s, lane);
        *reinterpret_cast<float2*>(A + (i0 + (m >> 2)) * LC_T + j0 + (m & 3)) = make_float2(s[0], s[1]);
    }
    __syncthreads();
    // ... and the halves: the last block's queries also take block 2's decays, the first block's keys block 1's
    for (int u = tid; u < 16 * D; u += LC_THREADS) {
        const int i = u / D, ch = u % D;
        qs[(48 + i) * D + ch] *= LC_G(2, ch);
        ks[i * D + (((ch >> 2) ^ (i & 7)) << 2) + (ch & 3)] *= LC_G(1, ch);
    }
    __syncthreads();
    {
        const int i0 = 32 + (lane & 28), j0 = 4 * warp;
        float s[16];
        lc_pairs<D, 4>(qs, ks, i0, j0, (lane & 3) + (lane & 4), s);
        const int m = lc_gather<16, 4>(s, lane);
        *reinterpret_cast<float4*>(A + (i0 + (m >> 2)) * LC_T + j0) = make_float4(s[0], s[1], s[2], s[3]);
    }
    __syncthreads();
    // queries times all decays from the chunk's start; the values over the keys
    for (int u = tid; u < 48 * D; u += LC_THREADS) {
        const int i = u / D, ch = u % D;
        const float g0 = LC_G(0, ch);
        qs[(16 + i) * D + ch] *= i < 16 ? g0 : g0 * LC_G(1, ch);
    }
#undef LC_G
    lc_load_values<DV>(p, ks, a0, nt, h);
    // o = q S + A V: four warps take one half of the channels and of the keys, four the other; a thread owns eight
    // tokens (eight apart, so that all have the same share of A's triangle) x 4 or 8 columns
    constexpr int NC = DV / 64, HD = D / 2, SLICES = HD / 8;
    constexpr int SL = LC_T * D / (16 * DV) < SLICES ? LC_T * D / (16 * DV) : SLICES;      // slices that as holds
    const int col = (tid & 15) * 4, half = tid >> 7, rg = (tid >> 4) & 7;
    const float* S = p.L + ((size_t)blockIdx.x * p.H + h) * p.d * p.dv;
    auto slice = [&](int s) {          // eight rows of S for either half, zeros behind d and dv
        if (s < SLICES) {
            float* dst = as + (s % SL) * 16 * DV;
#pragma unroll
            for (int it = 0; it < 16 * DV / 4 / LC_THREADS; ++it) {
                const int i = tid + it * LC_THREADS, rr = i / (DV / 4), cc = (i % (DV / 4)) * 4;
                const int row = (rr >> 3) * HD + 8 * s + (rr & 7);
                const bool ok = row < p.d && cc < p.dv;
                lc_fetch(dst + i * 4, ok ? S + (size_t)row * p.dv + cc : S, ok);
            }
        }
        lc_commit();
    };
    float4 acc[8][NC];
#pragma unroll
    for (int m = 0; m < 8; ++m)
#pragma unroll
        for (int x = 0; x < NC; ++x) acc[m][x] = f4(0.f);
#pragma unroll
    for (int s = 0; s < SL - 1; ++s) slice(s);
#pragma unroll 1
    for (int s = 0; s < SLICES; ++s) {
        lc_wait<SL - 2>();             // slice s (and the values, issued before it) is here
        __syncthreads();               // ... for all threads, and slice s - 1 is done with
        slice(s + SL - 1);
        const float* Ss = as + (s % SL) * 16 * DV + half * 8 * DV + col;
        const float* qr = qs + rg * D + half * HD + 8 * s;
#pragma unroll 1
        for (int cc = 0; cc < 8; cc += 2) {
            float4 sv[2][NC];
#pragma unroll
            for (int e = 0; e < 2; ++e)
#pragma unroll
                for (int x = 0; x < NC; ++x) sv[e][x] = *reinterpret_cast<const float4*>(Ss + (cc + e) * DV + x * 64);
#pragma unroll
            for (int m = 0; m < 8; ++m) {
                const float2 qq = *reinterpret_cast<const float2*>(qr + 8 * m * D + cc);
#pragma unroll
                for (int x = 0; x < NC; ++x) {
                    fma4(acc[m][x], qq.x, sv[0][x]);
                    fma4(acc[m][x], qq.y, sv[1][x]);
                }
            }
        }
    }
#pragma unroll 1
    for (int jj = 0; jj < 32; jj += 2) {               // keys jj of the half: four of every eight
        const int jb = jj >> 2, j = jb * 8 + half * 4 + (jj & 3);
        float4 vv[2][NC];
#pragma unroll
        for (int e = 0; e < 2; ++e)
#pragma unroll
            for (int x = 0; x < NC; ++x) vv[e][x] = *reinterpret_cast<const float4*>(ks + (j + e) * DV + x * 64 + col);
#pragma unroll
        for (int m = 0; m < 8; ++m) {
            if (m < jb) continue;
            const float2 w = *reinterpret_cast<const float2*>(A + (rg + 8 * m) * LC_T + j);
            // a value behind the query is left out, not multiplied by 0: it may be an infinity
            const bool sees = m > jb || j <= rg + 8 * m, next = m > jb || j + 1 <= rg + 8 * m;
#pragma unroll
            for (int x = 0; x < NC; ++x) {
                if (sees) fma4(acc[m][x], w.x, vv[0][x]);
                if (next) fma4(acc[m][x], w.y, vv[1][x]);
            }
        }
    }
    __syncthreads();
    // the halves' sums: each hands over four of its eight tokens (the place of queries and keys is free)
    float4* hand = reinterpret_cast<float4*>(qs);
#pragma unroll
    for (int m = 0; m < 4; ++m)
#pragma unroll
        for (int x = 0; x < NC; ++x) hand[(m * NC + x) * LC_THREADS + tid] = half ? acc[m][x] : acc[4 + m][x];
    __syncthreads();
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const int t = rg + 8 * (half * 4 + m);
#pragma unroll
        for (int x = 0; x < NC; ++x) {
            const float4 o = hand[(m * NC + x) * LC_THREADS + (tid ^ 128)], a = half ? acc[4 + m][x] : acc[m][x];
            if (t < nt && x * 64 + col < p.dv)
                *reinterpret_cast<float4*>(p.out + ((a0 + t) * p.all_heads + h) * p.dv + x * 64 + col) =
                    make_float4(p.q_scale * (a.x + o.x), p.q_scale * (a.y + o.y), p.q_scale * (a.z + o.z), p.q_scale * (a.w + o.w));
        }
    }
}

template <int D, int DV>
static int lc_go(const LcArgs& p, int n_portions, int n_chunks, cudaStream_t st) {
    constexpr int KD = D > DV ? D : DV;
    const size_t sm_chunk = (size_t)LC_T * (2 * D + DV) * 4, sm_out = (size_t)LC_T * (2 * D + KD + LC_T) * 4;
    cudaError_t e = cudaFuncSetAttribute(lc_chunk_kernel<D, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_chunk);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(lc_out_kernel<D, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_out);
    if (e != cudaSuccess) return (int)e;
    lc_chunk_kernel<D, DV><<<dim3(n_chunks, p.H), LC_THREADS, sm_chunk, st>>>(p);
    lc_scan_kernel<<<dim3((p.d * p.dv / 4 + LC_THREADS - 1) / LC_THREADS, n_portions * p.H), LC_THREADS, 0, st>>>(p);
    lc_out_kernel<D, DV><<<dim3(n_chunks, p.H), LC_THREADS, sm_out, st>>>(p);
    AIE_LAUNCH_CHECK();
}

// The arguments are those of aie_linear_recurrence.  Heads head0 .. head0 + heads - 1 of the H are done; L [n_chunks, heads, d, dv]
// and G [n_chunks, heads, d] float32 are scratch;
// n_portions, n_chunks: the requests that bring min_len tokens or more (the others are left alone), and their chunks of 64.
// Takes d and dv up to 128 in steps of 4 whose rows start on 16 bytes (else AIE_UNSUPPORTED: the caller takes the
// token-by-token kernel).
extern "C" int aie_linear_recurrence_chunked(const float* q, const float* k, const float* v, int ld, const float* decay_tok,
                                             int ld_decay, const float* decay_head, float q_scale, float k_scale, float* state,
                                             float* out, float* L, float* G, const int* q_start, const int* q_len, const int* slots,
                                             int R, int H, int head0, int heads, int d, int dv, int max_slots, int min_len, int n_portions,
                                             int n_chunks, const float* fg_lower, const float* fg_bias, unsigned* err, cudaStream_t st) {
    if (R <= 0 || n_portions <= 0 || n_chunks <= 0) return 0;
    if (heads <= 0 || head0 < 0 || head0 + heads > H || d <= 0 || dv <= 0 || min_len < 1 || (!decay_tok && !decay_head)) return AIE_BAD_ARG;
    if (fg_lower ? (!decay_tok || k) : !k) return AIE_BAD_ARG;
    const size_t at = (size_t)q | (size_t)k | (size_t)v | (size_t)decay_tok | (size_t)state | (size_t)out | (size_t)L |
                      (size_t)fg_lower | (size_t)fg_bias;
    if (d > 128 || dv > 128 || d % 4 || dv % 4 || ld % 4 || (decay_tok && ld_decay % 4) || (at & 15) ||
        heads > 65535 || (long long)n_portions * heads > 65535)
        return AIE_UNSUPPORTED;
    const size_t c = (size_t)head0 * d, cv = (size_t)head0 * dv;
    const auto from = [](const float* x, size_t n) { return x ? x + n : x; };
    const LcArgs p = {q + c, from(k, c), v + cv, from(decay_tok, c), from(decay_head, head0), from(fg_lower, c), from(fg_bias, c),
                      state + c * dv, out + cv, L, G, q_start, q_len, slots, err, ld, ld_decay, heads, H, R, d, dv, max_slots, min_len, q_scale, k_scale};
    if (d <= 64) return dv <= 64 ? lc_go<64, 64>(p, n_portions, n_chunks, st) : lc_go<64, 128>(p, n_portions, n_chunks, st);
    return dv <= 64 ? lc_go<128, 64>(p, n_portions, n_chunks, st) : lc_go<128, 128>(p, n_portions, n_chunks, st);
}
