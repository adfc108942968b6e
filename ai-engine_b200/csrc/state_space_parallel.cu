// The scalar-decay state-space recurrence of prompt portions, parallel over chunks of 64 tokens (the formulas are those of
// state_space_chunked.cu, whose blocks walk a request's chunks one behind the other and take 4.6 us a chunk; here the chain
// from chunk to chunk is a multiply-add an element):
//   chunk:  L_c = B^T (w * X),  w_s = exp(l_Q - l_s) dt_s, and the chunk's decay exp(l_Q), every (chunk, head) on its own
//   scan:   S_c+1 = exp(l_Q) S_c + L_c over a request's chunks, every element on its own; L_c is replaced by S_c
//   out:    Y = exp(l_t) (C S_c) + W X + skip X,  W[t, s] = (C_t . B_s) exp(l_t - l_s) dt_s   (s <= t)
// Operands, terms and sums are those of the other kernel: C, B and x enter rounded to bfloat16, w * X, W and the state as
// pairs of bfloat16 values, sums are float32.  Products run on mma.sync: a chunk's tiles are 64 x 64, W is made in the
// registers that the scores come in and meets X from there.  Bound by the traffic of the states (32 KB a chunk and head
// of 128 x 64, written, read, written and read again).  2,048 tokens x 64 heads in eight groups: 35 + 17 + 62 us, walked 260 us;
// 45 + 18 + 69 when results went four bytes at a time, the first warp made each head's decays while the others waited and the next
// head's state was asked for only when it was wanted; then with a head a block, which reads B and C anew, 46 + 18 + 80 us.
#include "attention_prefill.cuh"
#include "chunk_find.cuh"

#define SP_T 64
#define SP_THREADS 256

struct SpArgs {
    const float *C, *B, *X, *dt_raw, *dt_bias, *a_log, *skip;
    float *state, *out, *L, *G;
    const int *q_start, *q_len, *slots;
    unsigned* err;
    int ld, ld_dt, R, H, all_heads, head0, N, dv, hpg, max_slots, min_len, vec;      // H: the heads of this launch, from head0 on
    int hpb;             // neighbouring heads of one group that a block takes one after the other: B and C are read once for them
};

// [64][W] floats of a chunk's rows (columns of `src` up to n, rows up to nt; zeros elsewhere) as bfloat16, rows W + 8 apart
template <int W>
__device__ __forceinline__ void sp_load(bf16* dst, const float* src, size_t ld, int nt, int n, bool vec) {
    if (vec) {
        constexpr int PER = SP_T * W / 4 / SP_THREADS;
        float4 v[PER];
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int i = threadIdx.x + it * SP_THREADS, t = i / (W / 4), c = (i % (W / 4)) * 4;
            v[it] = t < nt && c < n ? *reinterpret_cast<const float4*>(src + t * ld + c) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int it = 0; it < PER; ++it) {
            const int i = threadIdx.x + it * SP_THREADS, t = i / (W / 4), c = (i % (W / 4)) * 4;
            *reinterpret_cast<uint2*>(dst + t * (W + 8) + c) = make_uint2(pack_bf16(v[it].x, v[it].y), pack_bf16(v[it].z, v[it].w));
        }
    } else {
        for (int i = threadIdx.x; i < SP_T * W; i += SP_THREADS) {
            const int t = i / W, c = i % W;
            dst[t * (W + 8) + c] = __float2bfloat16_rn(t < nt && c < n ? src[t * ld + c] : 0.f);
        }
    }
}

// step sizes and running sums of the log decays of a chunk's tokens (a token behind the end: no step, no decay) for the block's
// heads, 64 floats each, a warp a head, to be followed by a barrier.  (By the first warp from head to head the others waited for it.)
#define SP_HEADS 4          // heads a block takes at most
__device__ __forceinline__ void sp_decays(const SpArgs& p, size_t a0, int nt, int h_first, float (*dts)[SP_T], float (*las)[SP_T]) {
    if ((int)threadIdx.x < 32 * p.hpb) {
        const int lane = threadIdx.x & 31, h = h_first + (threadIdx.x >> 5);
        float *dt = dts[threadIdx.x >> 5], *la = las[threadIdx.x >> 5];
        const float rate = expf(p.a_log[h]), bias = p.dt_bias[h];
        float d[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            d[i] = 0.f;
            if (2 * lane + i < nt) {
                const float x = p.dt_raw[(a0 + 2 * lane + i) * p.ld_dt + h] + bias;
                d[i] = x > 20.f ? x : log1pf(expf(x));
            }
            dt[2 * lane + i] = d[i];
        }
        const float v0 = -rate * d[0], v1 = -rate * d[1];
        float run = v0 + v1;
        for (int o = 1; o < 32; o <<= 1) {
            const float up = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += up;
        }
        la[2 * lane] = run - v1;
        la[2 * lane + 1] = run;
    }
}
__device__ __forceinline__ void sp_split(float a, float b, unsigned& hi, unsigned& lo) {
    hi = pack_bf16(a, b);
    const float2 f = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&hi));
    lo = pack_bf16(a - f.x, b - f.y);
}

__device__ __forceinline__ void sp_copy(float* dst, const float* src, bool ok) {      // 16 bytes; zeros when not ok
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((unsigned)__cvta_generic_to_shared(dst)), "l"(src), "r"(ok ? 16 : 0) : "memory");
}

template <int NP>      // rows of the state, padded (zero rows change nothing); four blocks an SM: with three a fifth slower
__global__ void __launch_bounds__(SP_THREADS, 4) sp_chunk_kernel(SpArgs p) {
    extern __shared__ __align__(16) unsigned char sp_sm[];
    __shared__ int found[2];
    __shared__ float dts[SP_HEADS][SP_T], las[SP_HEADS][SP_T];
    constexpr int LN = NP + 8, LD = 64 + 8;
    bf16* Bs = reinterpret_cast<bf16*>(sp_sm);         // [64][NP]
    bf16* XH = Bs + SP_T * LN;                         // [64][64] x, then w * X, rounded
    bf16* XL = XH + SP_T * LD;                         //          ... and the rest
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h_first = blockIdx.y * p.hpb, col0 = blockIdx.z * 64;
    int r, c;
    chunk_find<SP_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(SP_T, p.q_len[r] - c * SP_T);
    const size_t a0 = (size_t)p.q_start[r] + c * SP_T;
    sp_decays(p, a0, nt, h_first, dts, las);
    sp_load<NP>(Bs, p.B + a0 * p.ld + (size_t)((p.head0 + h_first) / p.hpg) * p.N, p.ld, nt, p.N, p.vec);
#pragma unroll 1
    for (int h = h_first; h < h_first + p.hpb; ++h) {
        if (h > h_first) __syncthreads();                  // the last head's values are done with
        sp_load<64>(XH, p.X + a0 * p.ld + (size_t)h * p.dv + col0, p.ld, nt, p.dv - col0, p.vec);
        __syncthreads();
        const float *dt = dts[h - h_first], *la = las[h - h_first];
        const float l_end = la[SP_T - 1];
        if (tid == 0 && blockIdx.z == 0) p.G[(size_t)blockIdx.x * p.H + h] = expf(l_end);
#pragma unroll
        for (int it = 0; it < SP_T * 32 / SP_THREADS; ++it) {
            const int i = tid + it * SP_THREADS, t = i >> 5, j = (i & 31) * 2;
            const float w = expf(l_end - la[t]) * dt[t];
            unsigned* xp = reinterpret_cast<unsigned*>(XH + t * LD + j);
            const float2 x = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(xp));
            unsigned hi, lo;
            sp_split(x.x * w, x.y * w, hi, lo);
            *xp = hi;
            *reinterpret_cast<unsigned*>(XL + t * LD + j) = lo;
        }
        __syncthreads();
        // a job: 16 rows of the state x 32 of its columns
        float* L = p.L + ((size_t)blockIdx.x * p.H + h) * p.N * p.dv;
        for (int job = warp; job < NP / 16 * 2; job += SP_THREADS / 32) {
            const int m0 = (job >> 1) * 16, n0 = (job & 1) * 32;
            float acc[4][4] = {};
#pragma unroll
            for (int k = 0; k < SP_T; k += 16) {
                unsigned a[4];
                // rows = tokens: (k 0-7, m 0-7), (k 0-7, m 8-15), (k 8-15, m 0-7), (k 8-15, m 8-15), transposed on the way
                ldsm_x4_t(a[0], a[1], a[2], a[3], Bs + (k + (lane & 7) + ((lane >> 4) << 3)) * LN + m0 + ((lane >> 3) & 1) * 8);
#pragma unroll
                for (int np = 0; np < 2; ++np) {
                    unsigned b0, b1, b2, b3;
                    const int at = (k + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + n0 + np * 16 + (lane >> 4) * 8;
                    ldsm_x4_t(b0, b1, b2, b3, XH + at);
                    mma16816(acc[2 * np], a, b0, b1);
                    mma16816(acc[2 * np + 1], a, b2, b3);
                    ldsm_x4_t(b0, b1, b2, b3, XL + at);
                    mma16816(acc[2 * np], a, b0, b1);
                    mma16816(acc[2 * np + 1], a, b2, b3);
                }
            }
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int n = m0 + (lane >> 2) + 8 * e, j = col0 + n0 + x * 8 + (lane & 3) * 2;
                    if (n >= p.N) continue;
                    if (p.vec) {
                        if (j < p.dv) *reinterpret_cast<float2*>(L + (size_t)n * p.dv + j) = make_float2(acc[x][2 * e], acc[x][2 * e + 1]);
                        continue;
                    }
                    if (j < p.dv) L[(size_t)n * p.dv + j] = acc[x][2 * e];
                    if (j + 1 < p.dv) L[(size_t)n * p.dv + j + 1] = acc[x][2 * e + 1];
                }
        }
    }
}

// A thread owns V neighbouring elements of a state; eight chunks' loads are in flight while the chain runs.
template <int V>
__global__ void __launch_bounds__(SP_THREADS) sp_scan_kernel(SpArgs p) {
    __shared__ int found[2];
    const int h = blockIdx.y % p.H;
    int r, first;
    portion_find<SP_T>(p.q_len, p.R, p.min_len, blockIdx.y / p.H, found, r, first);
    if (r < 0) return;
    const int n = chunk_count<SP_T>(p.q_len, p.R, p.min_len, r), slot = p.slots[r];
    if (slot < 0 || slot >= p.max_slots) {
        if (threadIdx.x == 0) atomicOr(p.err, AIE_DEV_SLOT_OOB);
        return;
    }
    const int size = p.N * p.dv, e = (blockIdx.x * SP_THREADS + threadIdx.x) * V;
    if (e >= size) return;
    float* sp = p.state + ((size_t)slot * p.all_heads + h) * size + e;
    float* L = p.L + ((size_t)first * p.H + h) * size + e;
    const float* G = p.G + (size_t)first * p.H + h;
    const size_t ls = (size_t)p.H * size;
    float S[V];
    if constexpr (V == 4) {
        const float4 x = *reinterpret_cast<const float4*>(sp);
        S[0] = x.x, S[1] = x.y, S[2] = x.z, S[3] = x.w;
    } else {
        S[0] = *sp;
    }
    for (int c = 0; c < n; c += 8) {
        float l[8][V], g[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < n) {
                if constexpr (V == 4) {
                    const float4 x = *reinterpret_cast<const float4*>(L + (c + i) * ls);
                    l[i][0] = x.x, l[i][1] = x.y, l[i][2] = x.z, l[i][3] = x.w;
                } else {
                    l[i][0] = L[(c + i) * ls];
                }
                g[i] = G[(size_t)(c + i) * p.H];
            }
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (c + i < n) {
                if constexpr (V == 4) *reinterpret_cast<float4*>(L + (c + i) * ls) = make_float4(S[0], S[1], S[2], S[3]);
                else L[(c + i) * ls] = S[0];
#pragma unroll
                for (int v = 0; v < V; ++v) S[v] = fmaf(g[i], S[v], l[i][v]);
            }
    }
    if constexpr (V == 4) *reinterpret_cast<float4*>(sp) = make_float4(S[0], S[1], S[2], S[3]);
    else *sp = S[0];
}

// Eight warps: 16 tokens x 32 of the block's 64 columns each (the scores are made for both halves of the columns).
template <int NP>
__global__ void __launch_bounds__(SP_THREADS, 2) sp_out_kernel(SpArgs p) {
    extern __shared__ __align__(16) unsigned char sp_sm[];
    __shared__ int found[2];
    __shared__ float dts[SP_HEADS][SP_T], las[SP_HEADS][SP_T];
    constexpr int LN = NP + 8, LD = 64 + 8;
    bf16* Cs = reinterpret_cast<bf16*>(sp_sm);         // [64][NP]
    bf16* Bs = Cs + SP_T * LN;                         // [64][NP]
    bf16* Xs = Bs + SP_T * LN;                         // [64][64]
    bf16* SH = Xs + SP_T * LD;                         // [NP][64]
    bf16* SL = SH + NP * LD;
    // with `vec` the next head's state (over C and B, which live in registers then) and values, as they are in memory
    float* St = reinterpret_cast<float*>(sp_sm);       // [NP][64]
    float* Xt = reinterpret_cast<float*>(SL + NP * LD);        // [64][64]
    static_assert(NP * 64 * 4 <= 2 * SP_T * LN * 2, "the state lies over C and B");
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h_first = blockIdx.y * p.hpb, col0 = blockIdx.z * 64;
    int r, c;
    chunk_find<SP_T>(p.q_len, p.R, p.min_len, blockIdx.x, found, r, c);
    if (r < 0) return;
    const int nt = min(SP_T, p.q_len[r] - c * SP_T);
    const size_t a0 = (size_t)p.q_start[r] + c * SP_T;
    sp_decays(p, a0, nt, h_first, dts, las);
    sp_load<NP>(Cs, p.C + a0 * p.ld + (size_t)((p.head0 + h_first) / p.hpg) * p.N, p.ld, nt, p.N, p.vec);
    sp_load<NP>(Bs, p.B + a0 * p.ld + (size_t)((p.head0 + h_first) / p.hpg) * p.N, p.ld, nt, p.N, p.vec);
    __syncthreads();
    const int ti = warp & 3, n0 = (warp >> 2) * 32, ta = ti * 16 + (lane >> 2), tb = ta + 8;
    unsigned cf[NP / 16][4];                           // the warp's 16 rows of C
#pragma unroll
    for (int k = 0; k < NP / 16; ++k)
        ldsm_x4(cf[k][0], cf[k][1], cf[k][2], cf[k][3], Cs + (ti * 16 + (lane & 15)) * LN + k * 16 + (lane >> 4) * 8);
    float g[4][2][4];                                  // C B^T of the warp's 16 tokens with 16 keys at a time
#pragma unroll
    for (int sj = 0; sj < 4; ++sj) {
#pragma unroll
        for (int x = 0; x < 4; ++x) g[sj][0][x] = g[sj][1][x] = 0.f;
        if (sj > ti) continue;
#pragma unroll
        for (int k = 0; k < NP / 16; ++k) {
            unsigned b0, b1, b2, b3;
            // rows = keys: (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, k 0-7), (keys 8-15, k 8-15)
            ldsm_x4(b0, b1, b2, b3, Bs + (sj * 16 + (lane & 7) + ((lane >> 4) << 3)) * LN + k * 16 + ((lane >> 3) & 1) * 8);
            mma16816(g[sj][0], cf[k], b0, b1);
            mma16816(g[sj][1], cf[k], b2, b3);
        }
    }
    auto fetch = [&](int h) {
        const float* S = p.L + ((size_t)blockIdx.x * p.H + h) * p.N * p.dv + col0;
        const float* X = p.X + a0 * p.ld + (size_t)h * p.dv + col0;
#pragma unroll
        for (int it = 0; it < NP * 16 / SP_THREADS; ++it) {
            const int i = tid + it * SP_THREADS, n = i >> 4, j = (i & 15) * 4;
            const bool ok = n < p.N && col0 + j < p.dv;
            sp_copy(St + i * 4, ok ? S + (size_t)n * p.dv + j : S, ok);
        }
#pragma unroll
        for (int it = 0; it < SP_T * 16 / SP_THREADS; ++it) {
            const int i = tid + it * SP_THREADS, t = i >> 4, j = (i & 15) * 4;
            const bool ok = t < nt && col0 + j < p.dv;
            sp_copy(Xt + i * 4, ok ? X + (size_t)t * p.ld + j : p.X, ok);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    if (p.vec) {
        __syncthreads();                                   // C and B are in registers
        fetch(h_first);
    }
#pragma unroll 1
    for (int h = h_first; h < h_first + p.hpb; ++h) {
        const float* S = p.L + ((size_t)blockIdx.x * p.H + h) * p.N * p.dv + col0;
        if (p.vec) {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();                               // ... for all threads, and the last head's operands are done with
#pragma unroll
            for (int it = 0; it < NP * 16 / SP_THREADS; ++it) {
                const int i = tid + it * SP_THREADS, n = i >> 4, j = (i & 15) * 4;
                const float4 v = *reinterpret_cast<const float4*>(St + i * 4);
                uint2 hi, lo;
                sp_split(v.x, v.y, hi.x, lo.x);
                sp_split(v.z, v.w, hi.y, lo.y);
                *reinterpret_cast<uint2*>(SH + n * LD + j) = hi;
                *reinterpret_cast<uint2*>(SL + n * LD + j) = lo;
            }
#pragma unroll
            for (int it = 0; it < SP_T * 16 / SP_THREADS; ++it) {
                const int i = tid + it * SP_THREADS, t = i >> 4, j = (i & 15) * 4;
                const float4 v = *reinterpret_cast<const float4*>(Xt + i * 4);
                *reinterpret_cast<uint2*>(Xs + t * LD + j) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
            }
        } else {
            if (h > h_first) __syncthreads();              // the last head's state and values are done with
            for (int i = tid; i < NP * 64; i += SP_THREADS) {
                const int n = i >> 6, j = i & 63;
                const float v = n < p.N && col0 + j < p.dv ? S[(size_t)n * p.dv + j] : 0.f;
                const bf16 hi = __float2bfloat16_rn(v);
                SH[n * LD + j] = hi;
                SL[n * LD + j] = __float2bfloat16_rn(v - __bfloat162float(hi));
            }
            sp_load<64>(Xs, p.X + a0 * p.ld + (size_t)h * p.dv + col0, p.ld, nt, p.dv - col0, false);
        }
        __syncthreads();
        if (p.vec && h + 1 < h_first + p.hpb) fetch(h + 1);      // lands while this head's products run
        const float *dt = dts[h - h_first], *la = las[h - h_first];
        const float lta = la[ta], ltb = la[tb];
        float y[4][4] = {};
#pragma unroll
        for (int k = 0; k < NP / 16; ++k)
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                unsigned b0, b1, b2, b3;
                const int at = (k * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + n0 + np * 16 + (lane >> 4) * 8;
                ldsm_x4_t(b0, b1, b2, b3, SH + at);
                mma16816(y[2 * np], cf[k], b0, b1);
                mma16816(y[2 * np + 1], cf[k], b2, b3);
                ldsm_x4_t(b0, b1, b2, b3, SL + at);
                mma16816(y[2 * np], cf[k], b0, b1);
                mma16816(y[2 * np + 1], cf[k], b2, b3);
            }
        const float ea = expf(lta), eb = expf(ltb);
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
            unsigned wh[4], wl[4];                         // W as the next product's operand: its registers are the scores'
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int s = sj * 16 + x * 8 + (lane & 3) * 2;
                const float l0 = la[s], l1 = la[s + 1], d0 = dt[s], d1 = dt[s + 1];
                sp_split(s <= ta ? g[sj][x][0] * __expf(lta - l0) * d0 : 0.f, s + 1 <= ta ? g[sj][x][1] * __expf(lta - l1) * d1 : 0.f, wh[2 * x], wl[2 * x]);
                sp_split(s <= tb ? g[sj][x][2] * __expf(ltb - l0) * d0 : 0.f, s + 1 <= tb ? g[sj][x][3] * __expf(ltb - l1) * d1 : 0.f, wh[2 * x + 1], wl[2 * x + 1]);
            }
#pragma unroll
            for (int np = 0; np < 2; ++np) {
                unsigned b0, b1, b2, b3;
                ldsm_x4_t(b0, b1, b2, b3, Xs + (sj * 16 + (lane & 7) + ((lane >> 3) & 1) * 8) * LD + n0 + np * 16 + (lane >> 4) * 8);
                mma16816(y[2 * np], wh, b0, b1);
                mma16816(y[2 * np + 1], wh, b2, b3);
                mma16816(y[2 * np], wl, b0, b1);
                mma16816(y[2 * np + 1], wl, b2, b3);
            }
        }
        const float sk = p.skip ? p.skip[h] : 0.f;
#pragma unroll
        for (int x = 0; x < 4; ++x)
#pragma unroll
            for (int e = 0; e < 2; ++e) {
                const int t = e ? tb : ta, j = n0 + x * 8 + (lane & 3) * 2;
                if (t >= nt) continue;
                float u = y[x][2 * e], v = y[x][2 * e + 1];
                if (p.skip) {
                    const float2 xs = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(Xs + t * LD + j));      // x as the products saw it
                    u = fmaf(sk, xs.x, u);
                    v = fmaf(sk, xs.y, v);
                }
                float* o = p.out + ((a0 + t) * p.all_heads + h) * p.dv + col0 + j;
                if (p.vec) {
                    if (col0 + j < p.dv) *reinterpret_cast<float2*>(o) = make_float2(u, v);
                    continue;
                }
                if (col0 + j < p.dv) o[0] = u;
                if (col0 + j + 1 < p.dv) o[1] = v;
            }
    }
}

template <int NP>
static int sp_go(const SpArgs& p, int n_portions, int n_chunks, cudaStream_t st) {
    const int LN = NP + 8, LD = 64 + 8;
    const size_t sm_chunk = (size_t)(SP_T * LN + 2 * SP_T * LD) * 2, sm_out = (size_t)(2 * SP_T * LN + SP_T * LD + 2 * NP * LD) * 2 + SP_T * 64 * 4;
    cudaError_t e = cudaFuncSetAttribute(sp_chunk_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_chunk);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(sp_out_kernel<NP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm_out);
    if (e != cudaSuccess) return (int)e;
    const dim3 grid(n_chunks, p.H / p.hpb, (p.dv + 63) / 64);
    const int size = p.N * p.dv;
    sp_chunk_kernel<NP><<<grid, SP_THREADS, sm_chunk, st>>>(p);
    if (size % 4 == 0 && !(((size_t)p.state | (size_t)p.L) & 15))
        sp_scan_kernel<4><<<dim3((size / 4 + SP_THREADS - 1) / SP_THREADS, n_portions * p.H), SP_THREADS, 0, st>>>(p);
    else
        sp_scan_kernel<1><<<dim3((size + SP_THREADS - 1) / SP_THREADS, n_portions * p.H), SP_THREADS, 0, st>>>(p);
    sp_out_kernel<NP><<<grid, SP_THREADS, sm_out, st>>>(p);
    AIE_LAUNCH_CHECK();
}

// The arguments are those of aie_state_space_chunked.  Heads head0 .. head0 + heads - 1 of the H are done; L [n_chunks, heads, N,
// dv] and G [n_chunks, heads] float32 are scratch;
// n_portions, n_chunks: the requests that bring min_len tokens or more (the others are left alone), and their chunks of 64.
// N <= 128.
extern "C" int aie_state_space_parallel(const float* C, const float* B, const float* X, int ld, const float* dt_raw, int ld_dt,
                                        const float* dt_bias, const float* a_log, const float* skip, float* state, float* out,
                                        float* L, float* G, const int* q_start, const int* q_len, const int* slots, int R, int H, int head0, int heads,
                                        int N, int dv, int hpg, int max_slots, int min_len, int n_portions, int n_chunks, unsigned* err,
                                        cudaStream_t st) {
    if (R <= 0 || n_portions <= 0 || n_chunks <= 0) return 0;
    if (heads <= 0 || head0 < 0 || head0 + heads > H || N <= 0 || dv <= 0 || hpg < 1 || H % hpg || !dt_raw || !dt_bias || !a_log || min_len < 1) return AIE_BAD_ARG;
    if (N > 128 || heads > 65535 || (long long)n_portions * heads > 65535 || (dv + 63) / 64 > 65535) return AIE_UNSUPPORTED;
    const int vec = N % 4 == 0 && dv % 4 == 0 && ld % 4 == 0 && !(((size_t)C | (size_t)B | (size_t)X | (size_t)L) & 15) && !((size_t)out & 7);
    // four or two heads a block where that still gives every SM's two places a block
    int hpb = 1;
    while (hpb < SP_HEADS && hpg % (2 * hpb) == 0 && head0 % (2 * hpb) == 0 && heads % (2 * hpb) == 0 &&
           (long long)n_chunks * (heads / (2 * hpb)) * ((dv + 63) / 64) >= 2 * aie_sm_count()) hpb *= 2;
    const size_t c = (size_t)head0 * dv;
    const SpArgs p = {C, B, X + c, dt_raw + head0, dt_bias + head0, a_log + head0, skip ? skip + head0 : skip, state + c * N, out + c, L, G,
                      q_start, q_len, slots, err, ld, ld_dt, R, heads, H, head0, N, dv, hpg, max_slots, min_len, vec, hpb};
    if (N <= 32) return sp_go<32>(p, n_portions, n_chunks, st);
    if (N <= 64) return sp_go<64>(p, n_portions, n_chunks, st);
    return sp_go<128>(p, n_portions, n_chunks, st);
}
