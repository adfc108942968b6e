// The gated delta rule of prompt portions with all of a chunk's work that does not need the state done for all chunks side by
// side (the formulas and symbols are those of delta_rule_chunked.cu, whose blocks do everything chunk after chunk, and the
// part that does not depend on the columns once for every block of columns: 11.5 us a chunk, 184 us for 1024 tokens of 16
// heads of 128 x 128).  With T = (I + A)^-1,
//     U = T (beta V) - T (beta exp(l) K) S_0 = U0 - W S_0
// so that three kernels do it, for those 1024 tokens in 26 + 29 + 23 us:
//   prepare  every (chunk, head): unit keys, A, T, U0 and W, the keys times exp(l_Q - l_s), the chunk's decay
//   walk     every (request, head, 16 or 32 columns): U = U0 - W S,  S <- exp(l_Q) S + (w K)^T U  from chunk to chunk; U takes
//            U0's place, the states that chunks start from are kept
//   out      every (chunk, head): O = exp(l_t) Q S_0 + P U
// The walk is the chain that bounds it, 1.8 us a chunk with 16 columns a block: two products, two barriers and the exchange of the
// state one after the other on eight warps an SM, no unit near its limit.  W, the keys and U0 lie in memory as the walk wants them
// in shared memory and come in three bulk copies a chunk, and what goes back goes 16 bytes a thread from shared memory: 16 bytes a
// thread through cp.async and four bytes at a time back it was 2.7 us (3.5 with 32 columns), a bulk copy a row 3.3.  Without any
// traffic 1.45.  W and keys straight from L2 to the registers of their products: 2.4 us.
// T is made in float32: diagonal blocks of 16 by forward substitution, what is below from them.  T, beta V and beta exp(l)
// enter the products of U0 and W as three bfloat16 values, all 24 bits; on the FMA units prepare took 39 us.  Everything else
// enters mma.sync as pairs of bfloat16 values, as before, with float32 sums; the products that the state or the output is summed
// from keep the product of the two rests too, which makes up for W's rounding (errors against 64 bits: of the outputs 0.85 to
// 0.91 times, of the states 0.76 to 0.84 times those of delta_rule_chunked.cu).  The state stays in the walking warps'
// accumulators.
#include "attention_prefill.cuh"
#include "chunk_find.cuh"
#include "tc_common.cuh"

#define DP_T 64
#define DP_THREADS 256
#define DP_E 128                    // value columns that `prepare` holds at a time

struct DpArgs {
    const float *q, *k, *v, *b_raw, *a_raw, *a_log, *dt_bias;
    float *state, *out;
    bf16 *W, *Kw;             // [n_chunks, H, 2][64][d]: rounded value, rest; eight columns j of row t at place j ^ (t & 7) (dp_at)
    float *U, *S0, *decay;    // [n_chunks, H][e / 16][64][16], [n_chunks, H][d][e], [n_chunks, H]
    const int *q_start, *q_len, *slots, *live;
    unsigned* err;
    int ld, ldb, lda, R, H, all_heads, head0, per, e, max_slots, min_len;      // H: the heads of this launch, from head0 on; per a q/k head
    float q_scale, unit_eps;
};

__device__ __forceinline__ void dp_split(float a, float b, unsigned& hi, unsigned& lo) {
    hi = pack_bf16(a, b);
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi));
    lo = pack_bf16(a - f.x, b - f.y);
}
// the same and the rest of the rest: all 24 bits of a mantissa
__device__ __forceinline__ void dp_split3(float a, float b, unsigned& hi, unsigned& lo, unsigned& tail) {
    dp_split(a, b, hi, lo);
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi)), g = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&lo));
    tail = pack_bf16((a - f.x) - g.x, (b - f.y) - g.y);
}
// where column c of row t of W and Kw lies: as in shared memory, so that a chunk's come in one copy and ldmatrix reads eight rows
// without conflicts
template <int D> __device__ __forceinline__ int dp_at(int t, int c) { return t * D + ((c & ~7) ^ ((t & 7) << 3)) + (c & 7); }
// from global to shared memory, both on 16 bytes; the bytes count on the barrier
__device__ __forceinline__ void dp_bulk(void* dst, const void* src, int bytes, unsigned long long* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                 ::"r"(tc_smem(dst)), "l"(src), "r"(bytes), "r"(tc_smem(bar)) : "memory");
}
// acc += (ah + al) (bh + bl) without al bl, which is as small as what the pairs leave out
__device__ __forceinline__ void dp_mma3(float* acc, const unsigned* ah, const unsigned* al, unsigned bh0, unsigned bh1, unsigned bl0, unsigned bl1) {
    mma16816(acc, ah, bh0, bh1);
    mma16816(acc, ah, bl0, bl1);
    mma16816(acc, al, bh0, bh1);
}

// The chunk's unit vectors (times `scale`) of x as pairs, rows D + 8 apart; a warp makes every eighth row, all loads first.
// Kw (optional): the pairs of the same times exp(l_end - la[t]), [2][64][D].
template <int D>
__device__ __forceinline__ void dp_units(const float* x, size_t ld, int nt, float eps, float scale, bf16* hi, bf16* lo, const float* la, bf16* Kw) {
    constexpr int V = D / 32, ROWS = DP_T / 8;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    float v[ROWS][V];
#pragma unroll
    for (int rr = 0; rr < ROWS; ++rr) {
        const int t = warp + rr * 8;
        if constexpr (V == 4) {
            const float4 y = t < nt ? *reinterpret_cast<const float4*>(x + t * ld + 4 * lane) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[rr][0] = y.x, v[rr][1] = y.y, v[rr][2] = y.z, v[rr][3] = y.w;
        } else {
            const float2 y = t < nt ? *reinterpret_cast<const float2*>(x + t * ld + 2 * lane) : make_float2(0.f, 0.f);
            v[rr][0] = y.x, v[rr][1] = y.y;
        }
    }
    if (Kw) __syncthreads();                           // la is there
#pragma unroll
    for (int rr = 0; rr < ROWS; ++rr) {
        const int t = warp + rr * 8;
        float ss = 0.f;
#pragma unroll
        for (int i = 0; i < V; ++i) ss += v[rr][i] * v[rr][i];
        const float inv = rsqrtf(warp_sum(ss) + eps) * scale, w = Kw ? expf(la[DP_T - 1] - la[t]) : 0.f;
#pragma unroll
        for (int i = 0; i < V; i += 2) {
            const float a = v[rr][i] * inv, b = v[rr][i + 1] * inv;
            unsigned h, l;
            dp_split(a, b, h, l);
            *reinterpret_cast<unsigned*>(hi + t * (D + 8) + V * lane + i) = h;
            *reinterpret_cast<unsigned*>(lo + t * (D + 8) + V * lane + i) = l;
            if (Kw) {
                dp_split(a * w, b * w, h, l);
                *reinterpret_cast<unsigned*>(Kw + dp_at<D>(t, V * lane + i)) = h;
                *reinterpret_cast<unsigned*>(Kw + DP_T * D + dp_at<D>(t, V * lane + i)) = l;
            }
        }
    }
}
// running sums of the log decays of a chunk's tokens and (optional) beta, by the first warp; to be followed by a barrier
__device__ __forceinline__ void dp_decays(const DpArgs& p, size_t a0, int nt, int h, float* la, float* be) {
    if (threadIdx.x >= 32) return;
    const int lane = threadIdx.x;
    const float rate = expf(p.a_log[h]), bias = p.dt_bias[h];
    float v[2];
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const int t = 2 * lane + i;
        float b = 0.f;
        v[i] = 0.f;                                    // a token behind the portion's end: no decay, no correction
        if (t < nt) {
            const float x = p.a_raw[(a0 + t) * p.lda + h] + bias;
            v[i] = -rate * (x > 20.f ? x : log1pf(expf(x)));
            if (be) b = 1.f / (1.f + expf(-p.b_raw[(a0 + t) * p.ldb + h]));
        }
        if (be) be[t] = b;
    }
    float run = v[0] + v[1];
    for (int o = 1; o < 32; o <<= 1) {
        const float up = __shfl_up_sync(0xffffffffu, run, o);
        if (lane >= o) run += up;
    }
    la[2 * lane] = run - v[1];
    la[2 * lane + 1] = run;
}

template <int D>
__global__ void __launch_bounds__(DP_THREADS, 2) dp_prepare_kernel(DpArgs p) {
    extern __shared__ __align__(16) unsigned char dp_sm[];
    __shared__ int found[2];
    __shared__ float la[DP_T], be[DP_T];
    constexpr int LN = D + 8, LA = DP_T + 4, LV = DP_E + 4;
    bf16* KH = reinterpret_cast<bf16*>(dp_sm);         // [64][LN] unit keys
    bf16* KL = KH + DP_T * LN;
    float* As = reinterpret_cast<float*>(KL + DP_T * LN);          // [64][LA]
    float* Ts = As + DP_T * LA;                        // [64][LA] the inverse, zeros above the diagonal
    float* Vf = Ts + DP_T * LA;                        // [64][LV] up to 128 columns of the values
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y;
    int r, c;
    chunk_find<DP_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(DP_T, p.q_len[r] - c * DP_T);
    const size_t a0 = (size_t)p.q_start[r] + c * DP_T, at = (size_t)blockIdx.x * p.H + h;
    auto values = [&](int c0) {                        // ahead of their use
        for (int i = tid; i < DP_T * DP_E / 4; i += DP_THREADS) {
            const int t = i / (DP_E / 4), j = (i % (DP_E / 4)) * 4;
            const bool ok = t < nt && c0 + j < p.e;
            cp_async16(Vf + t * LV + j, ok ? p.v + (a0 + t) * p.ld + (size_t)h * p.e + c0 + j : p.v, ok);
        }
        cp_async_commit();
    };
    values(0);
    dp_decays(p, a0, nt, h, la, be);
    for (int i = tid; i < DP_T * LA; i += DP_THREADS) Ts[i] = 0.f;
    dp_units<D>(p.k + a0 * p.ld + (size_t)((p.head0 + h) / p.per) * D, p.ld, nt, p.unit_eps, 1.f, KH, KL, la, p.Kw + at * 2 * DP_T * D);
    __syncthreads();
    if (tid == 0) p.decay[at] = expf(la[DP_T - 1]);
    // A on and below the diagonal, tiles of 16 x 16 (1/0, ... as the warps come by them)
    for (int job = warp; job < 10; job += 8) {
        const int ti = job < 1 ? 0 : (job < 3 ? 1 : (job < 6 ? 2 : 3)), tj = job - ti * (ti + 1) / 2;
        float acc[2][4] = {};
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            unsigned ah[4], al[4], b[4], l[4];
            const int aat = (ti * 16 + (lane & 15)) * LN + k * 16 + (lane >> 4) * 8;
            const int bat = (tj * 16 + (lane & 7) + ((lane >> 4) << 3)) * LN + k * 16 + ((lane >> 3) & 1) * 8;
            ldsm_x4(ah[0], ah[1], ah[2], ah[3], KH + aat);
            ldsm_x4(al[0], al[1], al[2], al[3], KL + aat);
            ldsm_x4(b[0], b[1], b[2], b[3], KH + bat);
            ldsm_x4(l[0], l[1], l[2], l[3], KL + bat);
            dp_mma3(acc[0], ah, al, b[0], b[1], l[0], l[1]);
            dp_mma3(acc[1], ah, al, b[2], b[3], l[2], l[3]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int t = ti * 16 + (lane >> 2) + (e >> 1) * 8, s = tj * 16 + x * 8 + (lane & 3) * 2 + (e & 1);
                As[t * LA + s] = s < t ? be[t] * __expf(la[t] - la[s]) * acc[x][e] : 0.f;
            }
    }
    __syncthreads();
    // diagonal blocks of T: a thread a column, forward substitution in registers
    if (tid < DP_T) {
        const int blk = tid >> 4, cc = tid & 15;
        const float* A = As + blk * 16 * LA + blk * 16;
        float m[16];
#pragma unroll
        for (int t = 0; t < 16; ++t) {
            float acc0 = t == cc ? 1.f : 0.f, acc1 = 0.f;
#pragma unroll
            for (int s = 0; s + 1 < t; s += 2) {
                acc0 -= A[t * LA + s] * m[s];
                acc1 -= A[t * LA + s + 1] * m[s + 1];
            }
            if (t & 1) acc0 -= A[t * LA + t - 1] * m[t - 1];
            m[t] = acc0 + acc1;
            Ts[(blk * 16 + t) * LA + blk * 16 + cc] = m[t];
        }
    }
    __syncthreads();
    // what is below them, first in blocks of 16, then the block of 32: T21 = -T22 (A21 T11); A21 T11 stands in T21's place
    {
        const int col = (tid & 3) * 4, row = (tid >> 2) & 15, o = (tid >> 6) * 32;       // the first 128 threads
        float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
        auto product = [&](const float* A, const float* B, int n) {
#pragma unroll 4
            for (int k = 0; k < n; k += 4) {
                const float4 a = *reinterpret_cast<const float4*>(A + k);
                const float m[4] = {a.x, a.y, a.z, a.w};
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 b = *reinterpret_cast<const float4*>(B + (k + i) * LA);
                    x = make_float4(fmaf(m[i], b.x, x.x), fmaf(m[i], b.y, x.y), fmaf(m[i], b.z, x.z), fmaf(m[i], b.w, x.w));
                }
            }
        };
        auto put = [&](float* at, float sign) { *reinterpret_cast<float4*>(at) = make_float4(sign * x.x, sign * x.y, sign * x.z, sign * x.w); };
        if (tid < 128) {
            product(As + (o + 16 + row) * LA + o, Ts + o * LA + o + col, 16);
            put(Ts + (o + 16 + row) * LA + o + col, 1.f);
        }
        __syncthreads();
        x = make_float4(0.f, 0.f, 0.f, 0.f);
        if (tid < 128) product(Ts + (o + 16 + row) * LA + o + 16, Ts + (o + 16) * LA + o + col, 16);
        __syncthreads();
        if (tid < 128) put(Ts + (o + 16 + row) * LA + o + col, -1.f);
        __syncthreads();
        const int col2 = (tid & 7) * 4, row2 = 32 + (tid >> 3);
        x = make_float4(0.f, 0.f, 0.f, 0.f);
        product(As + row2 * LA, Ts + col2, 32);
        put(Ts + row2 * LA + col2, 1.f);
        __syncthreads();
        x = make_float4(0.f, 0.f, 0.f, 0.f);
        product(Ts + row2 * LA + 32, Ts + 32 * LA + col2, 32);
        __syncthreads();
        put(Ts + row2 * LA + col2, -1.f);
        cp_async_wait<0>();
        __syncthreads();
    }
    // W = (T beta exp(l)) K and U0 = (T beta) V: a warp 16 tokens x half of the columns; T's pairs are made in registers
    const int ti = warp & 3, half = warp >> 2, ta = ti * 16 + (lane >> 2), sc = (lane & 3) * 2;
    unsigned th[4][4], tl[4][4], tt[4][4];
    auto pairs = [&](bool keys) {
#pragma unroll
        for (int sj = 0; sj < 4; ++sj) {
            if (sj > ti) continue;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int s = sj * 16 + sc + (i >> 1) * 8;
                const float2 x = *reinterpret_cast<const float2*>(Ts + (ta + (i & 1) * 8) * LA + s);
                float w0 = be[s], w1 = be[s + 1];
                if (keys) w0 *= expf(la[s]), w1 *= expf(la[s + 1]);
                dp_split3(x.x * w0, x.y * w1, th[sj][i], tl[sj][i], tt[sj][i]);
            }
        }
    };
    pairs(true);
#pragma unroll 1
    for (int n0 = half * (D / 2); n0 < (half + 1) * (D / 2); n0 += 16) {
        float g[2][4] = {};
#pragma unroll
        for (int sj = 0; sj < 4; ++sj) {
            if (sj > ti) continue;
            const int bat = (sj * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LN + n0 + (lane >> 4) * 8;
            unsigned b[4], l[4];
            ldsm_x4_t(b[0], b[1], b[2], b[3], KH + bat);
            ldsm_x4_t(l[0], l[1], l[2], l[3], KL + bat);
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                dp_mma3(g[x], th[sj], tl[sj], b[2 * x], b[2 * x + 1], l[2 * x], l[2 * x + 1]);
                mma16816(g[x], tl[sj], l[2 * x], l[2 * x + 1]);
                mma16816(g[x], tt[sj], b[2 * x], b[2 * x + 1]);
            }
        }
#pragma unroll
        for (int x = 0; x < 2; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                unsigned hi, lo;
                dp_split(g[x][2 * y], g[x][2 * y + 1], hi, lo);
                bf16* w = p.W + at * 2 * DP_T * D + dp_at<D>(ta + 8 * y, n0 + x * 8 + sc);
                *reinterpret_cast<unsigned*>(w) = hi;
                *reinterpret_cast<unsigned*>(w + DP_T * D) = lo;
            }
    }
    pairs(false);
#pragma unroll 1
    for (int c0 = 0; c0 < p.e; c0 += DP_E) {
        if (c0) {
            __syncthreads();                           // the last columns are done with
            values(c0);
            cp_async_wait<0>();
            __syncthreads();
        }
        const int cols = min(DP_E, p.e - c0), per = (cols / 8 + 1) / 2 * 8;      // the first half's columns
#pragma unroll 1
        for (int n0 = half * per; n0 < min(cols, (half + 1) * per); n0 += 8) {
            float g[4] = {};
#pragma unroll
            for (int sj = 0; sj < 4; ++sj) {
                if (sj > ti) continue;
                const float* B = Vf + (sj * 16 + sc) * LV + n0 + (lane >> 2);
                unsigned b0, b1, l0, l1, t0, t1;
                dp_split3(B[0], B[LV], b0, l0, t0);
                dp_split3(B[8 * LV], B[9 * LV], b1, l1, t1);
                dp_mma3(g, th[sj], tl[sj], b0, b1, l0, l1);
                mma16816(g, tl[sj], l0, l1);
                mma16816(g, th[sj], t0, t1);
                mma16816(g, tt[sj], b0, b1);
            }
            float* u = p.U + at * DP_T * p.e + (size_t)((c0 + n0) / 16 * DP_T + ta) * 16 + (n0 & 8) + sc;
            *reinterpret_cast<float2*>(u) = make_float2(g[0], g[1]);
            *reinterpret_cast<float2*>(u + 8 * 16) = make_float2(g[2], g[3]);
        }
    }
}

// From chunk to chunk.  Eight warps: U in tiles of 16 tokens x DV / 2 columns; the state in D / 16 tiles of 16 rows x DV columns,
// float32 in its warp's accumulators, as pairs in shared memory for the next chunk.  The next chunk's W and keys are on
// their way meanwhile.  The wait for them is bounded (see tc_common.cuh): a block that gives up leaves the request's state as it was.
#ifndef DP_STRAY          // bytes that a chunk's barrier waits for beyond those that come: for the test of a wait that runs out
#define DP_STRAY 0
#endif
template <int D, int DV>
__global__ void __launch_bounds__(DP_THREADS, 1) dp_walk_kernel(DpArgs p) {
    extern __shared__ __align__(16) unsigned char dp_sm[];
    constexpr int LD = DV + 8, ST = 4 * DP_T * D, NU = DV / 16, NS = DV / 8;
    bf16* stage = reinterpret_cast<bf16*>(dp_sm);      // two of [WH | WL | KH | KL], each [64][D] (dp_at)
    bf16* SH = stage + 2 * ST;                         // [D][LD]
    bf16* SL = SH + D * LD;
    bf16* UH = SL + D * LD;                            // [64][LD]
    bf16* UL = UH + DP_T * LD;
    float* Us = reinterpret_cast<float*>(UL + DP_T * LD);          // two of [DV / 16][64][16]: U0
    __shared__ unsigned long long bars[2];             // a chunk's operands have landed
    __shared__ int gave_up;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, col0 = blockIdx.x * DV, h = blockIdx.y;
    __shared__ int found[2];
    int r, first;
    portion_find<DP_T>(p.q_len, p.R, p.min_len, blockIdx.z, found, r, first);
    if (r < 0) return;
    const int n = chunk_count<DP_T>(p.q_len, p.R, p.min_len, r), slot = p.slots[r];
    if (slot < 0 || slot >= p.max_slots) {
        if (tid == 0) atomicOr(p.err, AIE_DEV_SLOT_OOB);
        return;
    }
    // A chunk's operands come in three bulk copies (16 bytes at a time through the load/store units they took 12 of 43 us, in a
    // bulk copy a row 53)
    auto fetch = [&](int c) {
        if (c >= n || tid != 0) return;
        const size_t at = (size_t)(first + c) * p.H + h;
        constexpr int PAIR = 2 * DP_T * D * 2, COLS = DP_T * DV * 4;
        unsigned long long* bar = &bars[c & 1];
        mbar_expect_tx(bar, 2 * PAIR + COLS + DP_STRAY);
        dp_bulk(stage + (c & 1) * ST, p.W + at * 2 * DP_T * D, PAIR, bar);
        dp_bulk(stage + (c & 1) * ST + 2 * DP_T * D, p.Kw + at * 2 * DP_T * D, PAIR, bar);
        dp_bulk(Us + (c & 1) * DP_T * DV, p.U + at * DP_T * p.e + (size_t)col0 * DP_T, COLS, bar);
    };
    if (tid == 0) {
        gave_up = 0;
        mbar_init(&bars[0], 1);
        mbar_init(&bars[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        fetch(0);
    }
    __syncthreads();
    // a matrix of pairs in shared memory to rows (`row` floats apart, groups of 16 columns `group` apart) that take the place of
    // float32 ones: 16 rounded values, their 16 rests, ...; 16 bytes a thread
    auto store = [&](float* dst, size_t row_step, size_t group_step, const bf16* hi, const bf16* lo, int rows) {
        for (int i = tid; i < rows * DV / 4; i += DP_THREADS) {
            const int row = i / (DV / 4), x = i % (DV / 4), j = (x >> 2) * 16;      // x & 3: the rounded ones' halves, the rests'
            *reinterpret_cast<uint4*>(dst + row * row_step + (x >> 2) * group_step + (x & 3) * 4) =
                *reinterpret_cast<const uint4*>((x & 2 ? lo : hi) + row * LD + j + (x & 1) * 8);
        }
    };
    float* sp = p.state + ((size_t)slot * p.all_heads + h) * D * p.e + col0;
    const bool holds = warp < D / 16;                  // rows 16 warp .. + 15 of the state
    const int sr = warp * 16 + (lane >> 2), sc = (lane & 3) * 2;
    float S[NS][4];
#pragma unroll
    for (int x = 0; x < NS; ++x)
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            const float2 v = holds ? *reinterpret_cast<const float2*>(sp + (size_t)(sr + 8 * y) * p.e + x * 8 + sc) : make_float2(0.f, 0.f);
            S[x][2 * y] = v.x, S[x][2 * y + 1] = v.y;
        }
    const int ut = (warp & 3) * 16 + (lane >> 2), un = (warp >> 2) * 8 * NU;
    float decay = p.decay[(size_t)first * p.H + h];      // of the chunk, loaded a chunk ahead
    for (int c = 0; c < n; ++c) {
        const size_t at = (size_t)(first + c) * p.H + h;
        float* U = p.U + at * DP_T * p.e + (size_t)col0 * DP_T;
        if (holds) {
#pragma unroll
            for (int x = 0; x < NS; ++x)
#pragma unroll
                for (int y = 0; y < 2; ++y) {
                    unsigned hi, lo;
                    dp_split(S[x][2 * y], S[x][2 * y + 1], hi, lo);
                    *reinterpret_cast<unsigned*>(SH + (sr + 8 * y) * LD + x * 8 + sc) = hi;
                    *reinterpret_cast<unsigned*>(SL + (sr + 8 * y) * LD + x * 8 + sc) = lo;
                }
        }
        const bool ok = mbar_wait(&bars[c & 1], (c >> 1) & 1, &gave_up, p.err);
        if (__syncthreads_or(!ok)) {                   // this chunk's operands and state are here; the last chunk is done with
            if (tid == 0) tc_drain(bars, 2, c + 1);
            __syncthreads();
            return;
        }
        fetch(c + 1);
        store(p.S0 + at * D * p.e + col0, p.e, 16, SH, SL, D);
        const bf16* WH = stage + (c & 1) * ST;
        float a[NU][4] = {}, ahl[NU][4] = {}, alh[NU][4] = {};     // three chains of products
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            unsigned ah[4], al[4];
            const int aat = dp_at<D>((warp & 3) * 16 + (lane & 15), k * 16 + (lane >> 4) * 8);
            ldsm_x4(ah[0], ah[1], ah[2], ah[3], WH + aat);
            ldsm_x4(al[0], al[1], al[2], al[3], WH + DP_T * D + aat);
            const int bat = (k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + un + (NU > 1 ? (lane >> 4) * 8 : 0);
            unsigned b[4], l[4];
            ldsm_x4_t(b[0], b[1], b[2], b[3], SH + bat);
            ldsm_x4_t(l[0], l[1], l[2], l[3], SL + bat);
#pragma unroll
            for (int x = 0; x < NU; ++x) {
                mma16816(a[x], ah, b[2 * x], b[2 * x + 1]);
                mma16816(ahl[x], ah, l[2 * x], l[2 * x + 1]);
                mma16816(alh[x], al, b[2 * x], b[2 * x + 1]);
                mma16816(ahl[x], al, l[2 * x], l[2 * x + 1]);
            }
        }
#pragma unroll
        for (int x = 0; x < NU; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                const float2 u0 = *reinterpret_cast<const float2*>(Us + (c & 1) * DP_T * DV + (((un + x * 8) >> 4) * DP_T + ut + 8 * y) * 16 + ((un + x * 8) & 8) + sc);
                const float v0 = u0.x - (a[x][2 * y] + (ahl[x][2 * y] + alh[x][2 * y]));
                const float v1 = u0.y - (a[x][2 * y + 1] + (ahl[x][2 * y + 1] + alh[x][2 * y + 1]));
                unsigned hi, lo;
                dp_split(v0, v1, hi, lo);
                *reinterpret_cast<unsigned*>(UH + (ut + 8 * y) * LD + un + x * 8 + sc) = hi;
                *reinterpret_cast<unsigned*>(UL + (ut + 8 * y) * LD + un + x * 8 + sc) = lo;
            }
        const float g = decay;
        if (c + 1 < n) decay = p.decay[at + p.H];
        __syncthreads();
        store(U, 16, DP_T * 16, UH, UL, DP_T);
        if (holds) {
            const bf16* KH = WH + 2 * DP_T * D;
#pragma unroll
            for (int x = 0; x < NS; ++x)
#pragma unroll
                for (int y = 0; y < 4; ++y) S[x][y] *= g;
#pragma unroll
            for (int k = 0; k < DP_T; k += 16) {
                unsigned ah[4], al[4];
                const int aat = dp_at<D>(k + (lane & 7) + ((lane >> 4) << 3), warp * 16 + ((lane >> 3) & 1) * 8);
                ldsm_x4_t(ah[0], ah[1], ah[2], ah[3], KH + aat);
                ldsm_x4_t(al[0], al[1], al[2], al[3], KH + DP_T * D + aat);
#pragma unroll
                for (int x = 0; x < NS; x += 2) {
                    const int bat = (k + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + x * 8 + (lane >> 4) * 8;
                    unsigned b[4], l[4];
                    ldsm_x4_t(b[0], b[1], b[2], b[3], UH + bat);
                    ldsm_x4_t(l[0], l[1], l[2], l[3], UL + bat);
#pragma unroll
                    for (int y = 0; y < 2; ++y) {
                        dp_mma3(S[x + y], ah, al, b[2 * y], b[2 * y + 1], l[2 * y], l[2 * y + 1]);
                        mma16816(S[x + y], al, l[2 * y], l[2 * y + 1]);
                    }
                }
            }
        }
    }
    if (holds && (p.live == nullptr || p.live[r] != 0)) {
#pragma unroll
        for (int x = 0; x < NS; ++x)
#pragma unroll
            for (int y = 0; y < 2; ++y)
                *reinterpret_cast<float2*>(sp + (size_t)(sr + 8 * y) * p.e + x * 8 + sc) = make_float2(S[x][2 * y], S[x][2 * y + 1]);
    }
}

// Eight warps: 16 tokens x 32 of 64 columns each, a block of columns after the other.
template <int D>
__global__ void __launch_bounds__(DP_THREADS, 2) dp_out_kernel(DpArgs p) {
    extern __shared__ __align__(16) unsigned char dp_sm[];
    __shared__ int found[2];
    __shared__ float la[DP_T];
    constexpr int LN = D + 8, LD = 64 + 8;
    bf16* QH = reinterpret_cast<bf16*>(dp_sm);         // [64][LN]
    bf16* QL = QH + DP_T * LN;
    bf16* KH = QL + DP_T * LN;                         // [64][LN], until the scores are made
    bf16* KL = KH + DP_T * LN;
    bf16* SH = KH;                                     // [D][LD]
    bf16* SL = SH + D * LD;
    bf16* UH = SL + D * LD;                            // [64][LD]
    bf16* UL = UH + DP_T * LD;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h = blockIdx.y, hq = (p.head0 + h) / p.per;
    int r, c;
    chunk_find<DP_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(DP_T, p.q_len[r] - c * DP_T);
    const size_t a0 = (size_t)p.q_start[r] + c * DP_T, at = (size_t)blockIdx.x * p.H + h;
    dp_units<D>(p.q + a0 * p.ld + (size_t)hq * D, p.ld, nt, p.unit_eps, p.q_scale, QH, QL, nullptr, nullptr);
    dp_units<D>(p.k + a0 * p.ld + (size_t)hq * D, p.ld, nt, p.unit_eps, 1.f, KH, KL, nullptr, nullptr);
    dp_decays(p, a0, nt, h, la, nullptr);
    __syncthreads();
    const int ti = warp & 3, n0 = (warp >> 2) * 32, ta = ti * 16 + (lane >> 2), tb = ta + 8;
    const float lta = la[ta], ltb = la[tb];
    unsigned ph[4][4], pl[4][4];                       // P as the next product's operand: its registers are the scores'
#pragma unroll
    for (int sj = 0; sj < 4; ++sj) {
        if (sj > ti) continue;
        float g[2][4] = {};
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            unsigned ah[4], al[4], b[4], l[4];
            const int aat = (ti * 16 + (lane & 15)) * LN + k * 16 + (lane >> 4) * 8;
            const int bat = (sj * 16 + (lane & 7) + ((lane >> 4) << 3)) * LN + k * 16 + ((lane >> 3) & 1) * 8;
            ldsm_x4(ah[0], ah[1], ah[2], ah[3], QH + aat);
            ldsm_x4(al[0], al[1], al[2], al[3], QL + aat);
            ldsm_x4(b[0], b[1], b[2], b[3], KH + bat);
            ldsm_x4(l[0], l[1], l[2], l[3], KL + bat);
            dp_mma3(g[0], ah, al, b[0], b[1], l[0], l[1]);
            dp_mma3(g[1], ah, al, b[2], b[3], l[2], l[3]);
        }
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int s = sj * 16 + x * 8 + (lane & 3) * 2;
            const float l0 = la[s], l1 = la[s + 1];
            dp_split(s <= ta ? g[x][0] * __expf(lta - l0) : 0.f, s + 1 <= ta ? g[x][1] * __expf(lta - l1) : 0.f, ph[sj][2 * x], pl[sj][2 * x]);
            dp_split(s <= tb ? g[x][2] * __expf(ltb - l0) : 0.f, s + 1 <= tb ? g[x][3] * __expf(ltb - l1) : 0.f, ph[sj][2 * x + 1], pl[sj][2 * x + 1]);
        }
    }
    const float ea = expf(lta), eb = expf(ltb);
#pragma unroll 1
    for (int col0 = 0; col0 < p.e; col0 += 64) {
        __syncthreads();                               // the last columns are done with
#pragma unroll
        for (int it = 0; it < (D + DP_T) * 16 / DP_THREADS; ++it) {
            const int i = tid + it * DP_THREADS, row = i >> 4, j = ((i >> 2) & 3) * 16;
            const bool state = row < D, rest = i & 2, ok = col0 + j < p.e;
            const int cj = ok ? col0 + j : 0;
            const float* src = (state ? p.S0 + (at * D + row) * p.e + cj : p.U + at * DP_T * p.e + (size_t)(cj / 16 * DP_T + row - D) * 16) + (i & 3) * 4;
            bf16* dst = (state ? (rest ? SL : SH) + row * LD : (rest ? UL : UH) + (row - D) * LD) + j + (i & 1) * 8;
            cp_async16(dst, src, ok);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();
        float y[4][4] = {};
#pragma unroll
        for (int k = 0; k < D / 16; ++k) {
            unsigned ah[4], al[4];
            const int aat = (ti * 16 + (lane & 15)) * LN + k * 16 + (lane >> 4) * 8;
            ldsm_x4(ah[0], ah[1], ah[2], ah[3], QH + aat);
            ldsm_x4(al[0], al[1], al[2], al[3], QL + aat);
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                const int bat = (k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + n0 + np * 16 + (lane >> 4) * 8;
                unsigned b[4], l[4];
                ldsm_x4_t(b[0], b[1], b[2], b[3], SH + bat);
                ldsm_x4_t(l[0], l[1], l[2], l[3], SL + bat);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    dp_mma3(y[2 * np + x], ah, al, b[2 * x], b[2 * x + 1], l[2 * x], l[2 * x + 1]);
                    mma16816(y[2 * np + x], al, l[2 * x], l[2 * x + 1]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            y[x][0] *= ea;
            y[x][1] *= ea;
            y[x][2] *= eb;
            y[x][3] *= eb;
        }
#pragma unroll
        for (int sj = 0; sj < 4; ++sj) {
            if (sj > ti) continue;
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                const int bat = (sj * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + n0 + np * 16 + (lane >> 4) * 8;
                unsigned b[4], l[4];
                ldsm_x4_t(b[0], b[1], b[2], b[3], UH + bat);
                ldsm_x4_t(l[0], l[1], l[2], l[3], UL + bat);
#pragma unroll
                for (int x = 0; x < 2; ++x) {
                    dp_mma3(y[2 * np + x], ph[sj], pl[sj], b[2 * x], b[2 * x + 1], l[2 * x], l[2 * x + 1]);
                    mma16816(y[2 * np + x], pl[sj], l[2 * x], l[2 * x + 1]);
                }
            }
        }
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = e ? tb : ta, j = col0 + n0 + x * 8 + (lane & 3) * 2;
                if (t < nt && j < p.e)
                    *reinterpret_cast<float2*>(p.out + ((a0 + t) * p.all_heads + h) * p.e + j) = make_float2(y[x][2 * e], y[x][2 * e + 1]);
            }
    }
}

template <int D>
static int dp_go(const DpArgs& p, int n_portions, int n_chunks, cudaStream_t st) {
    constexpr int LN = D + 8, LA = DP_T + 4;
    const size_t sm_prep = (size_t)2 * DP_T * LN * 2 + (size_t)(2 * DP_T * LA + DP_T * (DP_E + 4)) * 4;
    const size_t sm_out = (size_t)(2 * DP_T * LN + 2 * max(DP_T * LN, (D + DP_T) * 72)) * 2;
    cudaError_t e = cudaFuncSetAttribute(dp_prepare_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_prep);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(dp_out_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_out);
    if (e != cudaSuccess) return (int)e;
    dp_prepare_kernel<D><<<dim3(n_chunks, p.H), DP_THREADS, sm_prep, st>>>(p);
    // 16 columns a block while all blocks run at once; 32 read W and the keys half as often
#define WALK(DV)                                                                                                        \
    {                                                                                                                   \
        const size_t sm = (size_t)(8 * DP_T * D + 2 * (D + DP_T) * (DV + 8)) * 2 + (size_t)2 * DP_T * DV * 4;           \
        e = cudaFuncSetAttribute(dp_walk_kernel<D, DV>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);          \
        if (e != cudaSuccess) return (int)e;                                                                            \
        dp_walk_kernel<D, DV><<<dim3(p.e / DV, p.H, n_portions), DP_THREADS, sm, st>>>(p);                                \
    }
    if (p.e % 32 || (long long)n_portions * p.H * (p.e / 16) <= aie_sm_count()) WALK(16) else WALK(32)
#undef WALK
    dp_out_kernel<D><<<dim3(n_chunks, p.H), DP_THREADS, sm_out, st>>>(p);
    AIE_LAUNCH_CHECK();
}

// The arguments are those of aie_delta_rule_chunked.  Heads head0 .. head0 + heads - 1 of the H are done; scratch: W and Kw
// [n_chunks, heads, 2, 64, d] bf16, U [n_chunks, heads, 64, e], S0 [n_chunks, heads, d, e] and decay [n_chunks, heads] float32; n_portions, n_chunks: the requests that bring
// min_len tokens or more, and their chunks of 64.  Takes d of 64 or 128 and e a multiple of 16, with rows that start on 16 bytes
// (else AIE_UNSUPPORTED).
extern "C" int aie_delta_rule_parallel(const float* q, const float* k, const float* v, int ld, const float* b_raw, int ldb,
                                       const float* a_raw, int lda, const float* a_log, const float* dt_bias, float q_scale,
                                       float unit_eps, float* state, float* out, void* W, void* Kw, float* U, float* S0, float* decay,
                                       const int* q_start, const int* q_len, const int* slots, const int* live, int R, int H, int head0,
                                       int heads, int G, int d, int e, int max_slots, int min_len, int n_portions, int n_chunks,
                                       unsigned* err, cudaStream_t st) {
    if (R <= 0 || n_portions <= 0 || n_chunks <= 0) return 0;
    if (heads <= 0 || head0 < 0 || head0 + heads > H || G <= 0 || H % G || d <= 0 || e <= 0 || min_len < 1) return AIE_BAD_ARG;
    const size_t at = (size_t)q | (size_t)k | (size_t)v | (size_t)state | (size_t)out | (size_t)W | (size_t)Kw | (size_t)U | (size_t)S0;
    if ((d != 64 && d != 128) || e % 16 || ld % 4 || (at & 15) || heads > 65535 || n_portions > 65535) return AIE_UNSUPPORTED;
    const size_t c = (size_t)head0 * e;
    const DpArgs p = {q, k, v + c, b_raw + head0, a_raw + head0, a_log + head0, dt_bias + head0, state + c * d, out + c, (bf16*)W,
                      (bf16*)Kw, U, S0, decay, q_start, q_len, slots, live, err, ld, ldb, lda, R, heads, H, head0, H / G, e, max_slots, min_len, q_scale, unit_eps};
    return d == 64 ? dp_go<64>(p, n_portions, n_chunks, st) : dp_go<128>(p, n_portions, n_chunks, st);
}
