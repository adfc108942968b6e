// Tensor-core attention over the compressed cache (bfloat16 rows [latent (rank) | rotated key part (rot)], one per
// token, shared by all heads): see latent_attention.cu for the formula.  All heads of a token multiply the same
// cache rows, so the heads are the rows of the products: four warps take one query token and a group of 16 heads
// (one m16 tile of mma.sync m16n8k16, bf16 in, float32 accumulate) and walk the token's visible keys in chunks
// of 64 that start at multiples of 64 of the absolute key position.  A CTA takes TQ = 4 consecutive tokens of a portion: they
// share the gathered cache rows, whose traffic from L2 bounds the kernel, and differ only in their masks.  (Lone tokens
// take latent_decode_kernel below.)
//
// Per chunk: the 64 cache rows are gathered page by page into shared memory by 16-byte cp.async copies (rows
// outside the mask or the block table are zero-filled, so a probability of 0 never meets an unwritten row);
// S = Q K^T with the chunk's keys split over the four warps; scores, mask, running maximum and sum in float32
// in shared memory (eight threads a row); O += P V with the latent's columns split over the four warps, V being
// the first `rank` columns of the same rows (ldmatrix.trans).  Where the portions are few, each token's
// chunks are cut into `splits` parts that run as CTAs of their own and leave (maximum, sum, unnormalised output) for a
// joining kernel.  Weights enter the product with the rows rounded to bfloat16 and are summed so, or (PAIR) as two
// bfloat16 terms each, 16 bits of mantissa, beside a float32 sum.  A sink (exp(sink[h]) in the denominator, nothing in the output) opens the running softmax of the first part.
#include "attention_prefill.cuh"
#include "tc_common.cuh"

#define LT_KEYS 64
#define LT_ROWS 16
#define LT_THREADS 128
#define LT_TOKENS 4

template <int CW, bool PAIR>      // latent columns per warp (rank = 4 CW); weights as two terms
__global__ void __launch_bounds__(LT_THREADS * LT_TOKENS)
latent_attention_tc_kernel(const float* __restrict__ q_full, const bf16* __restrict__ pages, bf16* __restrict__ out,
                           float* __restrict__ part_o, float* __restrict__ part_ml, const int* __restrict__ tiles,
                           const int* __restrict__ q_start, const int* __restrict__ q_len,
                           const int* __restrict__ ctx_len, const int* __restrict__ block_table, int bt_width,
                           int num_pages, int P, int H, int dk, int window, float scale, int splits,
                           const float* __restrict__ sink, unsigned* err) {
    constexpr int RANK = 4 * CW, NT = CW / 8, TQ = LT_TOKENS, THREADS = LT_THREADS * TQ;
    extern __shared__ __align__(16) unsigned char lt_raw[];
    const int SK = dk + 8;                                        // padded row: ldmatrix rows fall on different banks
    bf16* q_all = reinterpret_cast<bf16*>(lt_raw);                // [TQ][16][SK]
    bf16* k_s = q_all + TQ * LT_ROWS * SK;                        // [64][SK]
    bf16* p_all = k_s + LT_KEYS * SK;                             // [TQ][16][64 + 8]
    constexpr int PR = TQ * LT_ROWS * (LT_KEYS + 8);              // with PAIR a second plane: what rounding p left out
    float* s_all = reinterpret_cast<float*>(p_all + (PAIR ? 2 : 1) * PR);              // [TQ][16][64 + 1]
    float* m_all = s_all + TQ * LT_ROWS * (LT_KEYS + 1);          // [TQ][16] running maximum
    float* l_all = m_all + TQ * LT_ROWS;                          // [TQ][16] running sum
    float* c_all = l_all + TQ * LT_ROWS;                          // [TQ][16] correction of this chunk

    pdl_launch_dependents();
    pdl_wait();
    const int row = tiles[2 * blockIdx.x], off = tiles[2 * blockIdx.x + 1];
    const int h0 = blockIdx.y * LT_ROWS, part = blockIdx.z;
    const int tid = threadIdx.x, tq = tid / LT_THREADS, ltid = tid % LT_THREADS, warp = (tid >> 5) & 3, lane = tid & 31;
    const int n_act = min(TQ, q_len[row] - off);                  // tokens of this CTA that exist
    const int pos_first = ctx_len[row] + off, pos_last = pos_first + n_act - 1;
    const int t = q_start[row] + off + tq;
    const bool active = tq < n_act;
    const int pos = active ? pos_first + tq : -1;                 // a token that does not exist sees no key
    int lo = 0, lo_first = 0;
    if (window > 0 && pos - window + 1 > 0) lo = pos - window + 1;
    if (window > 0 && pos_first - window + 1 > 0) lo_first = pos_first - window + 1;
    const int first_chunk = lo_first / LT_KEYS, n_chunks = pos_last / LT_KEYS - first_chunk + 1;
    const int per = (n_chunks + splits - 1) / splits;
    const int c_begin = first_chunk + part * per, c_end = min(first_chunk + n_chunks, c_begin + per);
    bf16* q_s = q_all + tq * LT_ROWS * SK;
    bf16* p_s = p_all + tq * LT_ROWS * (LT_KEYS + 8);
    float* s_s = s_all + tq * LT_ROWS * (LT_KEYS + 1);
    float* m_s = m_all + tq * LT_ROWS;
    float* l_s = l_all + tq * LT_ROWS;
    float* c_s = c_all + tq * LT_ROWS;

    // the 16 heads' queries, rounded to bfloat16 (rows past the last head are zero)
    for (int r = warp; r < LT_ROWS; r += 4) {                     // a warp converts whole rows, four elements a lane
        const bool on = active && h0 + r < H;
        const float* src = q_full + ((size_t)t * H + h0 + r) * dk;
        for (int c = lane * 4; c < dk; c += 128) {
            const float4 v = on ? *reinterpret_cast<const float4*>(src + c) : make_float4(0.f, 0.f, 0.f, 0.f);
            *reinterpret_cast<uint2*>(q_s + r * SK + c) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
        }
    }
    if (ltid < LT_ROWS) {
        const bool leaks = sink && part == 0 && h0 + ltid < H;
        m_s[ltid] = leaks ? sink[h0 + ltid] : -INFINITY;
        l_s[ltid] = leaks ? 1.f : 0.f;
    }
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const int pieces = dk / 8;                                    // 16-byte pieces a row

    for (int ch = c_begin; ch < c_end; ++ch) {
        const int k0 = ch * LT_KEYS;
        __syncthreads();                                          // the previous chunk's rows and probabilities are done with
        // a warp copies whole rows: one look-up of the page per row, the lanes take the row's 16-byte pieces
        for (int j = tid >> 5; j < LT_KEYS; j += THREADS / 32) {
            const int kp = k0 + j;
            bool ok = kp >= lo_first && kp <= pos_last;
            const bf16* src = pages;
            if (ok) {
                const int pidx = kp / P;
                const int page = pidx < bt_width ? block_table[(size_t)row * bt_width + pidx] : -1;
                if (page < 0 || page >= num_pages) {
                    if (lane == 0) atomicOr(err, AIE_DEV_PAGE_OOB);
                    ok = false;
                } else {
                    src = pages + ((size_t)page * P + (kp - pidx * P)) * dk;
                }
            }
            for (int c = lane; c < pieces; c += 32) cp_async16(k_s + j * SK + c * 8, ok ? src + c * 8 : pages, ok);
        }
        cp_async_commit();
        cp_async_wait<0>();
        __syncthreads();

        // S = Q K^T: warp w multiplies keys 16 w .. 16 w + 15
        // two sets of accumulators take alternate k steps, so that a product does not wait for the one before it
        // and the fragments of the next step are on their way while this step multiplies
        float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        float s2[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
        const bf16* qa = q_s + (lane & 15) * SK + (lane >> 4) * 8;
        // rows = keys; matrices: (keys 0-7, k 0-7), (keys 0-7, k 8-15), (keys 8-15, k 0-7), (keys 8-15, k 8-15)
        const bf16* kb = k_s + (warp * 16 + (lane & 7) + ((lane >> 4) << 3)) * SK + ((lane >> 3) & 1) * 8;
        int kk = 0;
#pragma unroll 2
        for (; kk + 32 <= dk; kk += 32) {
            unsigned a[4], c[4], b0, b1, b2, b3, d0, d1, d2, d3;
            ldsm_x4(a[0], a[1], a[2], a[3], qa + kk);
            ldsm_x4(b0, b1, b2, b3, kb + kk);
            ldsm_x4(c[0], c[1], c[2], c[3], qa + kk + 16);
            ldsm_x4(d0, d1, d2, d3, kb + kk + 16);
            mma16816(s[0], a, b0, b1);
            mma16816(s[1], a, b2, b3);
            mma16816(s2[0], c, d0, d1);
            mma16816(s2[1], c, d2, d3);
        }
        if (kk < dk) {
            unsigned a[4], b0, b1, b2, b3;
            ldsm_x4(a[0], a[1], a[2], a[3], qa + kk);
            ldsm_x4(b0, b1, b2, b3, kb + kk);
            mma16816(s[0], a, b0, b1);
            mma16816(s[1], a, b2, b3);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            s[0][e] += s2[0][e];
            s[1][e] += s2[1][e];
        }
#pragma unroll
        for (int nt = 0; nt < 2; ++nt) {
            const int col = warp * 16 + nt * 8 + (lane & 3) * 2, r0 = lane >> 2;
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int r = r0 + (e >> 1) * 8, c = col + (e & 1), kp = k0 + c;
                s_s[r * (LT_KEYS + 1) + c] = (kp >= lo && kp <= pos) ? s[nt][e] * scale : -INFINITY;
            }
        }
        __syncthreads();
        // running softmax: eight threads a row, eight keys a thread
        {
            const int r = ltid >> 3, g = ltid & 7;
            float v[8], mx = -INFINITY;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                v[i] = s_s[r * (LT_KEYS + 1) + g * 8 + i];
                mx = fmaxf(mx, v[i]);
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
            const float m_old = m_s[r], m_new = fmaxf(m_old, mx);
            float sum = 0.f;
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const float p = (m_new == -INFINITY || v[i] == -INFINITY) ? 0.f : expf(v[i] - m_new);
                const bf16 pb = __float2bfloat16_rn(p);
                p_s[r * (LT_KEYS + 8) + g * 8 + i] = pb;
                if (PAIR) p_s[PR + r * (LT_KEYS + 8) + g * 8 + i] = __float2bfloat16_rn(p - __bfloat162float(pb));
                sum += PAIR ? p : __bfloat162float(pb);          // the sum of what the product will multiply
            }
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
            __syncwarp();
            if (g == 0) {
                const float corr = (m_old == -INFINITY) ? 0.f : expf(m_old - m_new);
                c_s[r] = corr;
                l_s[r] = l_s[r] * corr + sum;
                m_s[r] = m_new;
            }
        }
        __syncthreads();
        // O = O * corr + P V: warp w owns latent columns CW w .. CW w + CW - 1
        {
            const float ca = c_s[lane >> 2], cb = c_s[(lane >> 2) + 8];
#pragma unroll
            for (int i = 0; i < NT; ++i) {
                acc[i][0] *= ca;
                acc[i][1] *= ca;
                acc[i][2] *= cb;
                acc[i][3] *= cb;
            }
#pragma unroll
            for (int kk = 0; kk < LT_KEYS; kk += 16) {
                unsigned a[4];
                ldsm_x4(a[0], a[1], a[2], a[3], p_s + (lane & 15) * (LT_KEYS + 8) + kk + (lane >> 4) * 8);
                unsigned a2[4];
                if (PAIR) ldsm_x4(a2[0], a2[1], a2[2], a2[3], p_s + PR + (lane & 15) * (LT_KEYS + 8) + kk + (lane >> 4) * 8);
#pragma unroll
                for (int np = 0; np < NT / 2; ++np) {
                    unsigned b0, b1, b2, b3;
                    // rows = keys kk .. kk + 15 of V; matrices: (k 0-7, n 0-7), (k 8-15, n 0-7), (k 0-7, n 8-15), (k 8-15, n 8-15)
                    ldsm_x4_t(b0, b1, b2, b3, k_s + (kk + (lane & 7) + ((lane >> 3) & 1) * 8) * SK + warp * CW + np * 16 + (lane >> 4) * 8);
                    mma16816(acc[2 * np], a, b0, b1);
                    mma16816(acc[2 * np + 1], a, b2, b3);
                    if (PAIR) {
                        mma16816(acc[2 * np], a2, b0, b1);
                        mma16816(acc[2 * np + 1], a2, b2, b3);
                    }
                }
            }
        }
    }
    __syncthreads();
    const int ra = lane >> 2, rb = ra + 8;
    if (!active) return;
    if (splits == 1) {
        const float ia = l_s[ra] > 0.f ? 1.0f / l_s[ra] : 0.f, ib = l_s[rb] > 0.f ? 1.0f / l_s[rb] : 0.f;
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int col = warp * CW + i * 8 + (lane & 3) * 2;
            if (h0 + ra < H)
                *reinterpret_cast<unsigned*>(out + ((size_t)t * H + h0 + ra) * RANK + col) = pack_bf16(acc[i][0] * ia, acc[i][1] * ia);
            if (h0 + rb < H)
                *reinterpret_cast<unsigned*>(out + ((size_t)t * H + h0 + rb) * RANK + col) = pack_bf16(acc[i][2] * ib, acc[i][3] * ib);
        }
    } else {
        // a part leaves its unnormalised output, maximum and sum (an empty part: sum 0)
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int col = warp * CW + i * 8 + (lane & 3) * 2;
            if (h0 + ra < H)
                *reinterpret_cast<float2*>(part_o + (((size_t)t * H + h0 + ra) * splits + part) * RANK + col) = make_float2(acc[i][0], acc[i][1]);
            if (h0 + rb < H)
                *reinterpret_cast<float2*>(part_o + (((size_t)t * H + h0 + rb) * splits + part) * RANK + col) = make_float2(acc[i][2], acc[i][3]);
        }
        if (ltid < LT_ROWS && h0 + ltid < H) {
            float* ml = part_ml + (((size_t)t * H + h0 + ltid) * splits + part) * 2;
            ml[0] = m_s[ltid];
            ml[1] = l_s[ltid];
        }
    }
}

// ---------------------------------------------------------------------------
// Requests that bring one token.  What bounds them is the stream of their cache rows, so the rows are cut evenly over the
// machine whatever the requests' lengths: the visible chunks of 32 keys of all such requests stand in one line, CTA i takes
// the i-th of gridDim.x equal stretches of it, and the rows of the next chunk are on their way, across the requests' ends,
// while a chunk is multiplied; two CTAs share an SM, so that one's chain of products and softmax fills the other's waits.  Eight warps
// multiply: the scores' products are split over four groups of eight keys and two halves of a row, the values' over eight ranges of
// the latent's columns.  A ninth looks the rows up, a lane a key, and asks for each with one bulk copy whose bytes count on the stage's
// barrier (rows that are not to be seen it fills with zeros): with 16-byte copies by the other eight, which all looked up the
// same places, four of five of their instructions were addresses.  A stretch that holds a whole
// request writes its result; others leave (maximum, sum, unnormalised output) in slot CTA + request for the join.
// 64 requests of 512 .. 4,096 keys, 16 heads, a latent of 512 (170 MB of rows, 26 us at the copy bandwidth): 47 us, 63 with the copies
// in the warps that multiply; 162 us with a CTA a (request, quarter of its keys) that loaded and multiplied in turn, 109 us with one
// CTA an SM and four chunks in flight, whose eight warps waited on one another.  Bound by the chain of a chunk's products, softmax and
// products.  Every wait is bounded (see tc_common.cuh).
#define LD_KEYS 32
#define LD_THREADS 256
#define LD_MIN_CHUNKS 2       // a stretch is at least this long: a CTA's start costs about as much as two chunks

__device__ __forceinline__ int ld_chunks(const int* q_len, const int* ctx_len, int R, int window, int r, int& first) {
    first = 0;
    if (r >= R || q_len[r] != 1) return 0;
    const int pos = ctx_len[r];
    first = (window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0) / LD_KEYS;
    return pos / LD_KEYS - first + 1;
}
// Chunks of all requests and the length of a stretch, by any whole warp.
__device__ __forceinline__ int ld_stretch(const int* q_len, const int* ctx_len, int R, int window, int G, int& total) {
    total = 0;
    int first;
    for (int base = 0; base < R; base += 32) total += ld_chunks(q_len, ctx_len, R, window, base + (threadIdx.x & 31), first);
    total = __reduce_add_sync(0xffffffffu, total);
    return max((total + G - 1) / G, LD_MIN_CHUNKS);
}

__device__ __forceinline__ void ld_sync() { asm volatile("barrier.sync 1, %0;\n" ::"n"(LD_THREADS) : "memory"); }
// the same, and whether any of the threads says so
__device__ __forceinline__ bool ld_sync_any(bool mine) {
    int any;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.ne.b32 p, %1, 0;\n\tbarrier.red.or.pred q, 1, %2, p;\n\tselp.b32 %0, 1, 0, q;\n\t}\n"
                 : "=r"(any) : "r"(mine ? 1 : 0), "n"(LD_THREADS) : "memory");
    return any != 0;
}

template <int NT, bool PAIR, int CTAS>     // NT: tiles of 8 latent columns a warp (rank = 64 NT); CTAS: blocks an SM
__global__ void __launch_bounds__(LD_THREADS + 32, CTAS)
latent_decode_kernel(const float* __restrict__ q_full, const bf16* __restrict__ pages, bf16* __restrict__ out,
                     float* __restrict__ part_o, float* __restrict__ part_ml, const int* __restrict__ q_start,
                     const int* __restrict__ q_len, const int* __restrict__ ctx_len, const int* __restrict__ block_table,
                     int bt_width, int num_pages, int P, int R, int H, int dk, int window, float scale,
                     const float* __restrict__ sink, unsigned* err) {
    constexpr int RANK = 64 * NT, SP = LD_KEYS + 8, SS = LD_KEYS + 2, NST = 2;
    extern __shared__ __align__(16) unsigned char lt_raw[];
    const int SK = dk + 8;
    bf16* q_s = reinterpret_cast<bf16*>(lt_raw);                  // [16][SK]
    bf16* k_s = q_s + LT_ROWS * SK;                               // [NST][32][SK]
    bf16* p_s = k_s + NST * LD_KEYS * SK + 32;                    // [1 or 2][16][SP] (32: what a last odd step reads past a row)
    float* s_s = reinterpret_cast<float*>(p_s + (PAIR ? 2 : 1) * LT_ROWS * SP);      // [2][16][SS]
    float* m_s = s_s + 2 * LT_ROWS * SS;                          // [16] running maximum, sum, correction
    float* l_s = m_s + LT_ROWS;
    float* c_s = l_s + LT_ROWS;
    __shared__ unsigned long long full[NST], empty[NST];
    __shared__ int abort_word, asked;                             // asked: chunks whose rows were asked for (see tc_drain)
    volatile int* abort_flag = &abort_word;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, h0 = blockIdx.y * LT_ROWS;
    if (tid == 0) {
        for (int i = 0; i < NST; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], LD_THREADS / 32);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    pdl_launch_dependents();
    pdl_wait();
    __syncthreads();
    int total, first;
    const int per = ld_stretch(q_len, ctx_len, R, window, gridDim.x, total);
    const int begin = blockIdx.x * per, cnt = min(total - begin, per);
    if (cnt <= 0) return;
    int r = 0, c = 0;                                             // request and chunk that the stretch starts in
    for (int base = 0, before = 0; base < R; base += 32) {
        const int m = ld_chunks(q_len, ctx_len, R, window, base + lane, first);
        int run = m;
        for (int o = 1; o < 32; o <<= 1) {
            const int up = __shfl_up_sync(0xffffffffu, run, o);
            if (lane >= o) run += up;
        }
        const unsigned hit = __ballot_sync(0xffffffffu, begin < before + run);
        if (hit) {
            const int l = __ffs(hit) - 1;
            r = base + l;
            c = begin - before - __shfl_sync(0xffffffffu, run - m, l);
            break;
        }
        before += __shfl_sync(0xffffffffu, run, 31);
    }
    if (warp == LD_THREADS / 32) {                                // the warp that asks for rows, a chunk ahead of the others
        int lr = r, lc = c, lfirst, ln = ld_chunks(q_len, ctx_len, R, window, r, lfirst);
        // lane l: place (page * P + offset) of key l of the chunk that is asked for next, -1: none or not to be seen
        auto places = [&](int i) {
            int at = -1;
            if (i < cnt) {
                const int pos = ctx_len[lr], kp = (lfirst + lc) * LD_KEYS + lane;
                if (kp <= pos && (window <= 0 || kp > pos - window)) {
                    const int pidx = kp / P, page = pidx < bt_width ? block_table[(size_t)lr * bt_width + pidx] : -1;
                    if (page < 0 || page >= num_pages) atomicOr(err, AIE_DEV_PAGE_OOB);
                    else at = page * P + (kp - pidx * P);
                }
                if (++lc == ln && i + 1 < cnt) {
                    lc = 0;
                    do ln = ld_chunks(q_len, ctx_len, R, window, ++lr, lfirst);
                    while (ln == 0 && lr < R);
                }
            }
            return at;
        };
        int at = places(0), i = 0;
        for (; i < cnt; ++i) {
            unsigned long long* bar = &full[i % NST];
            bool ok = true;
            if (i >= NST) ok = mbar_wait(&empty[i % NST], (i / NST - 1) & 1, abort_flag, err);
            if (!__all_sync(0xffffffffu, ok)) break;
            bf16* dst = k_s + ((i % NST) * LD_KEYS + lane) * SK;
            if (at < 0)
                for (int x = 0; x < dk; x += 8) *reinterpret_cast<uint4*>(dst + x) = make_uint4(0, 0, 0, 0);
            asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // (a later copy may land on such a row)
            const int rows = __popc(__ballot_sync(0xffffffffu, at >= 0));
            __syncwarp();                                         // lane 0's arrival publishes all lanes' zeros: a vote orders no memory
            if (lane == 0) mbar_expect_tx(bar, rows * dk * 2);
            __syncwarp();
            if (at >= 0)
                asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n"
                             ::"r"(tc_smem(dst)), "l"(pages + (size_t)at * dk), "r"(dk * 2), "r"(tc_smem(bar)) : "memory");
            at = places(i + 1);
        }
        if (lane == 0) asked = i;
    } else {
        const int steps = dk / 16, kg = warp & 3, kh = warp >> 2;
        const int step0 = kh ? (steps + 1) / 2 : 0, step1 = kh ? steps : (steps + 1) / 2;
        float acc[NT][4];
        int n = 0, c_begin = 0, pos = 0, lo = 0;
        bool fresh = true;
        for (int i = 0; i < cnt; ++i) {
            if (fresh) {                                              // a request begins: its queries, an empty softmax
                fresh = false;
                n = ld_chunks(q_len, ctx_len, R, window, r, first);
                c_begin = c;
                pos = ctx_len[r];
                lo = window > 0 ? max(pos - window + 1, 0) : 0;
                if (i > 0) ld_sync();                                 // the last one's sums have been read
                const int t = q_start[r];
                for (int rr = warp; rr < LT_ROWS; rr += LD_THREADS / 32) {
                    const bool on = h0 + rr < H;
                    const float* src = q_full + ((size_t)t * H + h0 + rr) * dk;
                    for (int x = lane * 4; x < dk; x += 128) {
                        const float4 v = on ? *reinterpret_cast<const float4*>(src + x) : make_float4(0.f, 0.f, 0.f, 0.f);
                        *reinterpret_cast<uint2*>(q_s + rr * SK + x) = make_uint2(pack_bf16(v.x, v.y), pack_bf16(v.z, v.w));
                    }
                }
                if (tid < LT_ROWS) {
                    const bool leaks = sink && c == 0 && h0 + tid < H;
                    m_s[tid] = leaks ? sink[h0 + tid] : -INFINITY;
                    l_s[tid] = leaks ? 1.f : 0.f;
                }
#pragma unroll
                for (int x = 0; x < NT; ++x) acc[x][0] = acc[x][1] = acc[x][2] = acc[x][3] = 0.f;
                ld_sync();
            }
            const bool ok = mbar_wait(&full[i % NST], (i / NST) & 1, abort_flag, err);
            __syncwarp();
            const bf16* ks = k_s + (i % NST) * LD_KEYS * SK;
            {
                float s0[4] = {0.f, 0.f, 0.f, 0.f}, s1[4] = {0.f, 0.f, 0.f, 0.f};
                const bf16* qa = q_s + (lane & 15) * SK + (lane >> 4) * 8;
                const bf16* kb = ks + (kg * 8 + (lane & 7)) * SK + (lane >> 3) * 8;
#pragma unroll 3
                for (int st = step0; st < step1; st += 2) {           // two steps of 16: one load of keys
                    unsigned a[4], b0, b1, b2, b3;
                    ldsm_x4(b0, b1, b2, b3, kb + st * 16);
                    ldsm_x4(a[0], a[1], a[2], a[3], qa + st * 16);
                    mma16816(s0, a, b0, b1);
                    if (st + 1 < step1) {
                        ldsm_x4(a[0], a[1], a[2], a[3], qa + st * 16 + 16);
                        mma16816(s1, a, b2, b3);
                    }
                }
                float* d = s_s + kh * LT_ROWS * SS + (lane >> 2) * SS + kg * 8 + (lane & 3) * 2;
                *reinterpret_cast<float2*>(d) = make_float2(s0[0] + s1[0], s0[1] + s1[1]);
                *reinterpret_cast<float2*>(d + 8 * SS) = make_float2(s0[2] + s1[2], s0[3] + s1[3]);
            }
            // all scores are there; nobody multiplies the weights and values of the chunk before any more
            if (ld_sync_any(!ok)) break;
            {                                                         // running softmax: sixteen threads a row, two keys a thread
                const int row = tid >> 4, g = tid & 15, key = (first + c) * LD_KEYS + 2 * g;
                const float2 x = *reinterpret_cast<const float2*>(s_s + row * SS + 2 * g);
                const float2 y = *reinterpret_cast<const float2*>(s_s + (LT_ROWS + row) * SS + 2 * g);
                const float v0 = key >= lo && key <= pos ? (x.x + y.x) * scale : -INFINITY;
                const float v1 = key + 1 >= lo && key + 1 <= pos ? (x.y + y.y) * scale : -INFINITY;
                float mx = fmaxf(v0, v1);
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xffffffffu, mx, o));
                const float m_old = m_s[row], m_new = fmaxf(m_old, mx);
                const float p0 = v0 == -INFINITY ? 0.f : expf(v0 - m_new), p1 = v1 == -INFINITY ? 0.f : expf(v1 - m_new);
                const unsigned pb = pack_bf16(p0, p1);
                const float2 pf = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&pb));
                *reinterpret_cast<unsigned*>(p_s + row * SP + 2 * g) = pb;
                if (PAIR) *reinterpret_cast<unsigned*>(p_s + (LT_ROWS + row) * SP + 2 * g) = pack_bf16(p0 - pf.x, p1 - pf.y);
                float sum = PAIR ? p0 + p1 : pf.x + pf.y;             // the sum of what the product will multiply
#pragma unroll
                for (int o = 8; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
                __syncwarp();
                if (g == 0) {
                    const float corr = m_old == -INFINITY ? 0.f : expf(m_old - m_new);
                    c_s[row] = corr;
                    l_s[row] = l_s[row] * corr + sum;
                    m_s[row] = m_new;
                }
            }
            ld_sync();
            {                                                         // O = O * corr + P V over this warp's columns
                const float ca = c_s[lane >> 2], cb = c_s[(lane >> 2) + 8];
#pragma unroll
                for (int x = 0; x < NT; ++x) {
                    acc[x][0] *= ca;
                    acc[x][1] *= ca;
                    acc[x][2] *= cb;
                    acc[x][3] *= cb;
                }
#pragma unroll
                for (int kk = 0; kk < LD_KEYS; kk += 16) {
                    unsigned a[4], a2[4];
                    ldsm_x4(a[0], a[1], a[2], a[3], p_s + (lane & 15) * SP + kk + (lane >> 4) * 8);
                    if (PAIR) ldsm_x4(a2[0], a2[1], a2[2], a2[3], p_s + LT_ROWS * SP + (lane & 15) * SP + kk + (lane >> 4) * 8);
                    const bf16* vb = ks + (kk + (lane & 7) + ((lane >> 3) & 1) * 8) * SK + warp * 8 * NT + (lane >> 4) * 8;
#pragma unroll
                    for (int np = 0; np < (NT + 1) / 2; ++np) {
                        unsigned b0, b1, b2, b3;
                        ldsm_x4_t(b0, b1, b2, b3, vb + np * 16);
                        mma16816(acc[2 * np], a, b0, b1);
                        if (2 * np + 1 < NT) mma16816(acc[2 * np + 1 < NT ? 2 * np + 1 : 0], a, b2, b3);
                        if (PAIR) {
                            mma16816(acc[2 * np], a2, b0, b1);
                            if (2 * np + 1 < NT) mma16816(acc[2 * np + 1 < NT ? 2 * np + 1 : 0], a2, b2, b3);
                        }
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_plain(&empty[i % NST]);
            ++c;
            if (c < n && i + 1 < cnt) continue;
            // the request, or the stretch, ends here
            const int ra = lane >> 2, rb = ra + 8, t = q_start[r];
            const bool whole = c_begin == 0 && c == n;
            const size_t slot = (size_t)(blockIdx.x + r) * H;
            const float ia = whole ? (l_s[ra] > 0.f ? 1.0f / l_s[ra] : 0.f) : 1.f, ib = whole ? (l_s[rb] > 0.f ? 1.0f / l_s[rb] : 0.f) : 1.f;
#pragma unroll
            for (int x = 0; x < NT; ++x) {
                const int col = warp * 8 * NT + x * 8 + (lane & 3) * 2;
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int hh = h0 + (e ? rb : ra);
                    if (hh >= H) continue;
                    const float u = acc[x][2 * e] * (e ? ib : ia), v = acc[x][2 * e + 1] * (e ? ib : ia);
                    if (whole) *reinterpret_cast<unsigned*>(out + ((size_t)t * H + hh) * RANK + col) = pack_bf16(u, v);
                    else *reinterpret_cast<float2*>(part_o + (slot + hh) * RANK + col) = make_float2(u, v);
                }
            }
            if (!whole && tid < LT_ROWS && h0 + tid < H) {
                part_ml[(slot + h0 + tid) * 2] = m_s[tid];
                part_ml[(slot + h0 + tid) * 2 + 1] = l_s[tid];
            }
            c = 0;
            fresh = true;
            if (i + 1 < cnt)
                do n = ld_chunks(q_len, ctx_len, R, window, ++r, first);
                while (n == 0 && r < R);
        }
    }
    __syncthreads();
    if (*abort_flag && tid == 0) tc_drain(full, NST, asked);
}

// One block a (request, head): the parts that the stretches of latent_decode_kernel left of it, in their order.
__global__ void __launch_bounds__(128)
latent_decode_join_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml, bf16* __restrict__ out,
                          const int* __restrict__ q_start, const int* __restrict__ q_len, const int* __restrict__ ctx_len, int R,
                          int H, int rank, int window, int G) {
    extern __shared__ float ld_w[];                               // [G] weights
    __shared__ int range_s[2];
    __shared__ float inv_s;
    pdl_launch_dependents();
    pdl_wait();
    const int r = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    if (q_len[r] != 1) return;
    if (tid < 32) {
        int total, first, start = 0;
        const int per = ld_stretch(q_len, ctx_len, R, window, G, total);
        for (int base = 0; base < r; base += 32) {
            const int i = base + tid;
            start += i < r ? ld_chunks(q_len, ctx_len, R, window, i, first) : 0;
        }
        start = __reduce_add_sync(0xffffffffu, start);
        const int p0 = start / per, p1 = (start + ld_chunks(q_len, ctx_len, R, window, r, first) - 1) / per;
        float mx = -INFINITY;
        for (int p = p0 + tid; p <= p1 && p1 > p0; p += 32) {
            const float* ml = part_ml + ((size_t)(p + r) * H + h) * 2;
            if (ml[1] > 0.f) mx = fmaxf(mx, ml[0]);
        }
        mx = warp_max(mx);
        float den = 0.f;
        for (int p = p0 + tid; p <= p1 && p1 > p0; p += 32) {
            const float* ml = part_ml + ((size_t)(p + r) * H + h) * 2;
            const float w = ml[1] > 0.f ? expf(ml[0] - mx) : 0.f;
            ld_w[p - p0] = w;
            den += w * ml[1];
        }
        den = warp_sum(den);
        if (tid == 0) {
            range_s[0] = p0;
            range_s[1] = p1;
            inv_s = den > 0.f ? 1.0f / den : 0.f;
        }
    }
    __syncthreads();
    const int p0 = range_s[0], parts = range_s[1] - p0 + 1;
    if (parts <= 1) return;                                       // one stretch held it whole
    for (int c = tid * 4; c < rank; c += blockDim.x * 4) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 4
        for (int p = 0; p < parts; ++p) {
            const float4 v = *reinterpret_cast<const float4*>(part_o + ((size_t)(p0 + p + r) * H + h) * rank + c);
            const float w = ld_w[p];
            acc = make_float4(fmaf(w, v.x, acc.x), fmaf(w, v.y, acc.y), fmaf(w, v.z, acc.z), fmaf(w, v.w, acc.w));
        }
        store4<bf16>(out + ((size_t)q_start[r] * H + h) * rank + c, make_float4(acc.x * inv_s, acc.y * inv_s, acc.z * inv_s, acc.w * inv_s));
    }
}

// The requests of the step that bring one token (the others are left alone).  q_full [T, H, dk] float32, pages [num_pages, P,
// dk] bfloat16, out [T, H, rank] bfloat16; part_o [G + R, H, rank] and part_ml [G + R, H, 2] float32 scratch.  rank = 64 ..
// 512 in steps of 64, dk a multiple of 16 up to 1,024 (else AIE_UNSUPPORTED).
extern "C" int aie_latent_decode(const float* q_full, const void* pages, void* out, float* part_o, float* part_ml,
                                 const int* q_start, const int* q_len, const int* ctx_len, const int* block_table, int bt_width,
                                 int num_pages, int P, int R, int H, int rank, int dk, int window, float scale, int G,
                                 const float* sink, int pair, unsigned* err, cudaStream_t st) {
    if (R <= 0) return 0;
    if (rank < 64 || rank > 512 || rank % 64 || dk % 16 || dk < rank || dk > 1024 || H <= 0) return AIE_UNSUPPORTED;
    if (G < 1 || G > 4096 || !part_o || !part_ml || P <= 0 || (long long)num_pages * P > 0x7fffffffLL) return AIE_BAD_ARG;
    if (((size_t)q_full | (size_t)pages) & 15) return AIE_BAD_ARG;      // (rows are copied from 16 bytes on)
    const dim3 grid(G, (H + LT_ROWS - 1) / LT_ROWS);
    if (grid.y > 65535 || H > 65535) return AIE_UNSUPPORTED;
    const size_t smem = (size_t)(LT_ROWS + 2 * LD_KEYS) * (dk + 8) * 2 + 64 + (size_t)(pair ? 2 : 1) * LT_ROWS * (LD_KEYS + 8) * 2 +
                        (size_t)(2 * LT_ROWS * (LD_KEYS + 2) + 3 * LT_ROWS) * 4;
    const bool two = 2 * (smem + 1024) <= (size_t)aie_smem_per_sm();      // rows of up to about 640 elements
    cudaError_t e = cudaSuccess;
#define GO2(NT, PV, CTAS)                                                                                               \
    {                                                                                                                   \
        auto kern = latent_decode_kernel<NT, PV, CTAS>;                                                                 \
        e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                         \
        if (e == cudaSuccess)                                                                                           \
            e = launch_pdl(kern, grid, dim3(LD_THREADS + 32), smem, st, q_full, (const bf16*)pages, (bf16*)out, part_o, part_ml, \
                           q_start, q_len, ctx_len, block_table, bt_width, num_pages, P, R, H, dk, window, scale, sink, err); \
    }
#define GO(NT)                                                                                                          \
    case NT:                                                                                                            \
        if (pair) { if (two) GO2(NT, true, 2) else GO2(NT, true, 1) }                                                   \
        else { if (two) GO2(NT, false, 2) else GO2(NT, false, 1) }                                                      \
        break;
    switch (rank / 64) {
        GO(1) GO(2) GO(3) GO(4) GO(5) GO(6) GO(7) GO(8)
        default: return AIE_UNSUPPORTED;
    }
#undef GO
#undef GO2
    if (e != cudaSuccess) return (int)e;
    launch_pdl(latent_decode_join_kernel, dim3(R, H), dim3(128), G * sizeof(float), st, part_o, part_ml, (bf16*)out, q_start, q_len,
               ctx_len, R, H, rank, window, G);
    AIE_LAUNCH_CHECK();
}

// out[t, h] = sum_p w_p O_p / sum_p w_p l_p with w_p = exp(m_p - max m), parts in order.  The first warp makes the
// weights of all parts (at most 64), then every thread adds its column with several parts' loads in flight.
__global__ void latent_join_kernel(const float* __restrict__ part_o, const float* __restrict__ part_ml,
                                   bf16* __restrict__ out, int splits, int rank) {
    __shared__ float w_s[64];
    __shared__ float inv_s;
    pdl_launch_dependents();
    pdl_wait();
    const size_t th = blockIdx.x;
    const float* ml = part_ml + th * splits * 2;
    if (threadIdx.x < 32) {
        const int a = threadIdx.x, b = a + 32;
        const float la = a < splits ? ml[2 * a + 1] : 0.f, lb = b < splits ? ml[2 * b + 1] : 0.f;
        const float ma = la > 0.f ? ml[2 * a] : -INFINITY, mb = lb > 0.f ? ml[2 * b] : -INFINITY;
        const float mx = warp_max(fmaxf(ma, mb));
        const float wa = la > 0.f ? expf(ma - mx) : 0.f, wb = lb > 0.f ? expf(mb - mx) : 0.f;
        w_s[a] = wa;
        w_s[b] = wb;
        const float den = warp_sum(wa * la + wb * lb);
        if (a == 0) inv_s = den > 0.f ? 1.0f / den : 0.f;
    }
    __syncthreads();
    const float inv = inv_s;
    for (int c = threadIdx.x * 4; c < rank; c += blockDim.x * 4) {
        float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll 8
        for (int p = 0; p < splits; ++p) {                 // an empty part wrote zeros and weighs nothing
            const float4 v = *reinterpret_cast<const float4*>(part_o + (th * splits + p) * rank + c);
            const float w = w_s[p];
            acc.x = fmaf(w, v.x, acc.x);
            acc.y = fmaf(w, v.y, acc.y);
            acc.z = fmaf(w, v.z, acc.z);
            acc.w = fmaf(w, v.w, acc.w);
        }
        store4<bf16>(out + th * rank + c, make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv));
    }
}

// q_full [T, H, dk] float32; pages [num_pages, P, dk] bfloat16; out [T, H, rank] bfloat16.  tiles [n_tiles, 2] =
// (request row, offset among the tokens it brings) of units of LT_TOKENS tokens; requests that it does not name are left
// alone.  Takes rank = 64 .. 512 in steps of 64, dk a multiple of 16 and rows that shared memory has room for (else
// AIE_UNSUPPORTED: the caller takes the plain kernel).  splits > 1 needs part_o [T, H, splits, rank] and part_ml [T, H,
// splits, 2] float32.
extern "C" int aie_latent_attention_tc(const float* q_full, const void* pages, void* out, float* part_o, float* part_ml,
                                       const int* tiles, int n_tiles, const int* q_start, const int* q_len,
                                       const int* ctx_len, const int* block_table, int bt_width,
                                       int num_pages, int P, int T, int H, int rank, int dk, int window, float scale,
                                       int splits, const float* sink, int pair, unsigned* err, cudaStream_t st) {
    if (T <= 0 || n_tiles <= 0) return 0;
    if (rank < 64 || rank > 512 || rank % 64 || dk % 16 || dk < rank || dk > 1024 || H <= 0) return AIE_UNSUPPORTED;
    if (splits < 1 || splits > 64 || (splits > 1 && (!part_o || !part_ml))) return AIE_BAD_ARG;
    const int SK = dk + 8;
    const size_t smem = (size_t)(LT_TOKENS * LT_ROWS + LT_KEYS) * SK * 2 + (size_t)LT_TOKENS * LT_ROWS * (LT_KEYS + 8) * 2 * (pair ? 2 : 1) +
                        (size_t)LT_TOKENS * (LT_ROWS * (LT_KEYS + 1) + 3 * LT_ROWS) * 4;
    if (smem > 220 * 1024) return AIE_UNSUPPORTED;
    dim3 grid(n_tiles, (H + LT_ROWS - 1) / LT_ROWS, splits);
    if (grid.y > 65535) return AIE_UNSUPPORTED;
#define GO1(CWV, PV)                                                                                                  \
    {                                                                                                                 \
        auto kern = latent_attention_tc_kernel<CWV, PV>;                                                              \
        cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);                           \
        launch_pdl(kern, grid, dim3(LT_THREADS * LT_TOKENS), smem, st, q_full, (const bf16*)pages, (bf16*)out, part_o, part_ml, tiles, \
                   q_start, q_len, ctx_len, block_table, bt_width, num_pages, P, H, dk, window, scale, splits, sink, err);             \
    }
#define GO(CWV)                                                                                                       \
    case CWV:                                                                                                         \
        if (pair) GO1(CWV, true) else GO1(CWV, false)                                                                 \
        break;
    switch (rank / 4) {
        GO(16) GO(32) GO(48) GO(64) GO(80) GO(96) GO(112) GO(128)
        default: return AIE_UNSUPPORTED;
    }
#undef GO
#undef GO1
#undef GO2
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return (int)e;
    if (splits > 1) launch_pdl(latent_join_kernel, dim3(T * H), dim3(128), 0, st, part_o, part_ml, (bf16*)out, splits, rank);
    AIE_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// Per-head products of small steps: out[t, h, n] = sum_k w[h, n, k] x[t, h, k], bfloat16 operands, float32 sums.  What
// bounds them is the stream of the weights.  A CTA of four warps owns 16 rows n of one head for all tokens; the warps
// take every fourth block of 32 k and are joined through shared memory.  A thread reads its operands 16 bytes at a
// time: the eight consecutive k it loads stand for the pairs that two mma.sync k16 steps want of it, in weights and
// activations alike, and a sum over k has no order to keep.
#define HL_TOKENS 64

template <int NT, typename O>       // token tiles of 8
__global__ void __launch_bounds__(128)
head_linear_small_kernel(const bf16* __restrict__ x, long long xt, long long xh, const bf16* __restrict__ w,
                         O* __restrict__ out, long long ot, long long oh, int T, int N, int K) {
    __shared__ float part[4][16][NT * 8 + 1];
    pdl_launch_dependents();
    pdl_wait();
    const int h = blockIdx.y, n0 = blockIdx.x * 16;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31, row = lane >> 2, q = lane & 3;
    const bf16* wh = w + (size_t)h * N * K;
    const bool on0 = n0 + row < N, on1 = n0 + row + 8 < N;
    const bf16* w0 = wh + (size_t)(on0 ? n0 + row : 0) * K + q * 8;
    const bf16* w1 = wh + (size_t)(on1 ? n0 + row + 8 : 0) * K + q * 8;
    float acc[NT][4];
#pragma unroll
    for (int i = 0; i < NT; ++i) acc[i][0] = acc[i][1] = acc[i][2] = acc[i][3] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
#pragma unroll 4
    for (int k = warp * 32; k < K; k += 128) {
        const uint4 a0 = on0 ? *reinterpret_cast<const uint4*>(w0 + k) : zero;
        const uint4 a1 = on1 ? *reinterpret_cast<const uint4*>(w1 + k) : zero;
        const unsigned f0[4] = {a0.x, a1.x, a0.y, a1.y}, f1[4] = {a0.z, a1.z, a0.w, a1.w};
#pragma unroll
        for (int i = 0; i < NT; ++i) {
            const int t = i * 8 + row;
            const uint4 b = t < T ? *reinterpret_cast<const uint4*>(x + t * xt + h * xh + k + q * 8) : zero;
            mma16816(acc[i], f0, b.x, b.y);
            mma16816(acc[i], f1, b.z, b.w);
        }
    }
#pragma unroll
    for (int i = 0; i < NT; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) part[warp][row + (e >> 1) * 8][i * 8 + q * 2 + (e & 1)] = acc[i][e];
    __syncthreads();
    for (int i = tid; i < 16 * NT * 8; i += 128) {
        const int n = i & 15, t = i >> 4;
        if (t < T && n0 + n < N)
            out[t * ot + h * oh + n0 + n] = from_f32<O>((part[0][n][t] + part[1][n][t]) + (part[2][n][t] + part[3][n][t]));
    }
}

// x rows xt apart (tokens) and xh apart (heads), out likewise (elements); w [H, N, K] bfloat16.  T <= 64, K a multiple of
// 32, x and its strides aligned to 16 bytes (else AIE_UNSUPPORTED).
extern "C" int aie_head_linear_small(const void* x, long long xt, long long xh, const void* w, void* out, int out_dtype,
                                     long long ot, long long oh, int T, int H, int N, int K, cudaStream_t st) {
    if (T <= 0) return 0;
    if (T > HL_TOKENS || K % 32 || xt % 8 || xh % 8 || ((size_t)x & 15) || ((size_t)w & 15) || H > 65535) return AIE_UNSUPPORTED;
    const dim3 grid((N + 15) / 16, H);
#define GO(NT, O) launch_pdl(head_linear_small_kernel<NT, O>, grid, dim3(128), 0, st, (const bf16*)x, xt, xh, (const bf16*)w, (O*)out, ot, oh, T, N, K)
#define GO_O(O)                                                                                                       \
    if (T <= 8) GO(1, O);                                                                                             \
    else if (T <= 16) GO(2, O);                                                                                       \
    else if (T <= 32) GO(4, O);                                                                                       \
    else GO(8, O)
    if (out_dtype == AIE_F32) {
        GO_O(float);
    } else if (out_dtype == AIE_BF16) {
        GO_O(bf16);
    } else {
        return AIE_BAD_ARG;
    }
#undef GO_O
#undef GO
    AIE_LAUNCH_CHECK();
}

// ---------------------------------------------------------------------------
// The cached rows that portions read expanded, one behind the other: tiles [n, 2] = (request row, which 128 keys of it counted
// from its first); rows before the window of the portion's first token or behind its last are zeros.  A block copies 8 rows
// of a tile, 16 bytes a thread (32 rows: 3,072 rows of 576 took 9.3 us in 96 blocks, now 5.3).
#define LG_ROWS 8
__global__ void __launch_bounds__(256)
latent_gather_kernel(const bf16* __restrict__ pages, bf16* __restrict__ rows, const int* __restrict__ tiles,
                     const int* __restrict__ q_len, const int* __restrict__ ctx_len, const int* __restrict__ block_table,
                     int bt_width, int num_pages, int P, int dk, int window, unsigned* err) {
    pdl_launch_dependents();
    pdl_wait();
    const int tile_i = blockIdx.x / (128 / LG_ROWS), sub = blockIdx.x % (128 / LG_ROWS), tid = threadIdx.x;
    const int r = tiles[2 * tile_i], key0 = tiles[2 * tile_i + 1] * 128 + sub * LG_ROWS, pieces = dk / 8;
    const int lo = window > 0 ? max(ctx_len[r] - window + 1, 0) : 0, last = ctx_len[r] + q_len[r] - 1;
    uint4* dst = reinterpret_cast<uint4*>(rows + ((size_t)tile_i * 128 + sub * LG_ROWS) * dk);
    for (int i = tid; i < LG_ROWS * pieces; i += 256) {
        const int key = key0 + i / pieces, c = i % pieces;
        uint4 v = make_uint4(0u, 0u, 0u, 0u);
        if (key >= lo && key <= last) {
            const int pidx = key / P, page = pidx < bt_width ? block_table[(size_t)r * bt_width + pidx] : -1;
            if (page < 0 || page >= num_pages) {
                if (c == 0) atomicOr(err, AIE_DEV_PAGE_OOB);
            } else {
                v = reinterpret_cast<const uint4*>(pages + ((size_t)page * P + (key - pidx * P)) * dk)[c];
            }
        }
        dst[i] = v;
    }
}

// pages [num_pages, P, dk] bf16, dk a multiple of 8; rows [n_tiles * 128, dk].
extern "C" int aie_latent_gather(const void* pages, void* rows, const int* tiles, int n_tiles, const int* q_len, const int* ctx_len,
                                 const int* block_table, int bt_width, int num_pages, int P, int dk, int window, unsigned* err,
                                 cudaStream_t st) {
    if (n_tiles <= 0) return 0;
    if (dk % 8 || P <= 0 || n_tiles > 0x1fffffff || (((size_t)pages | (size_t)rows) & 15)) return AIE_BAD_ARG;
    launch_pdl(latent_gather_kernel, dim3((unsigned)n_tiles * (128 / LG_ROWS)), dim3(256), 0, st, (const bf16*)pages, (bf16*)rows, tiles,
               q_len, ctx_len, block_table, bt_width, num_pages, P, dk, window, err);
    AIE_LAUNCH_CHECK();
}
