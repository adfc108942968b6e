// Attention over a compressed cache: per token the cache holds one latent vector c [rank] (shared by all
// heads, normalised) and one rotated key part kr [rot] (shared by all heads), together one row of
// dk = rank + rot elements.  A head's key is [W_uk c | kr] and its value W_uv c; with the up-projections
// folded into the query (qa = W_uk^T q_plain) and applied to the output (o = W_uv (sum_j p_j c_j)) the
// kernel reads the cache rows as they are: score_j = (qa . c_j + q_rot . kr_j) * scale, one "kv head" for all
// query heads.
//
// latent_prepare (q_plain with q_full, and q_all, may be left out: null): from the fused projection [q heads | c | kr] of the step's tokens it writes the plain
//   query parts (compute dtype, for the folding product), the rotated query parts (float32), in q_all both parts side by
//   side (compute dtype, for queries that meet expanded keys; with short_row [T] a token whose entry is >= 0 has the first two,
//   in that row, and the others have the last), and the
//   normalised c and rotated kr into the token's cache row.  The rotation pairs element 2i with 2i+1 over the
//   first `rot_dims` elements of the rot-wide part (or, with `halves`, element i with i + rot_dims / 2); the
//   angle is float(position) * inv_freq[i] in float32, and cosine and sine are multiplied by `mag`.  The latent and the key part may come from a projection
//   of their own (`kv`, rows ld_kv floats apart) when the queries are made by a second product.
// latent_attention: one block per (token, head); keys in chunks of 128 that start at multiples of 128 of the
//   absolute key position with a running maximum and sum, so a row's additions depend on its position only.
//   `sink` (a number per head, or null): exp(sink[h]) joins the denominator and adds nothing to the output.
#include "common.cuh"

#define LAT_CHUNK 128
#define LAT_PREP 128       // threads that share the sum over a latent

#define LAT_ANGLES 128     // angles a token that fit the table below (a rotation over up to 256 elements)

__device__ __forceinline__ float2 latent_angle(int pos, float freq, float mag) {
    float sn, cs;
    sincosf((float)pos * freq, &sn, &cs);
    return make_float2(cs * mag, sn * mag);
}

// element i of a rot-wide vector x after the rotation by `pos`; tab: the token's cosines and sines, or null
__device__ __forceinline__ float latent_rotated(const float* x, int i, int half, int halves, int pos,
                                                const float* __restrict__ inv_freq, float mag, const float2* tab) {
    if (i >= 2 * half) return x[i];
    const int j = halves ? (i < half ? i : i - half) : i >> 1;
    const float2 a = tab ? tab[j] : latent_angle(pos, inv_freq[j], mag);
    if (halves) return i < half ? x[i] * a.x - x[i + half] * a.y : x[i] * a.x + x[j] * a.y;
    return (i & 1) ? x[i] * a.x + x[i - 1] * a.y : x[i] * a.x - x[i + 1] * a.y;
}

template <typename A, typename C>
__global__ void latent_prepare_kernel(const float* __restrict__ proj, int ld, int H, int d, int rot, int rank,
                                      int rot_dims, int has_kv, const float* __restrict__ c_weight, float eps,
                                      const float* __restrict__ inv_freq, A* __restrict__ q_plain,
                                      float* __restrict__ q_full, C* __restrict__ pages,
                                      const int* __restrict__ positions, const int* __restrict__ token_req,
                                      const int* __restrict__ block_table, int bt_width, int num_pages, int P,
                                      unsigned* err, const float* __restrict__ kv, int ld_kv, int halves, float mag,
                                      A* __restrict__ q_all, const int* __restrict__ short_row) {
    __shared__ float red[32];
    __shared__ float2 angles[LAT_ANGLES];              // made once a token, for all heads
    pdl_launch_dependents();
    pdl_wait();
    const int t = blockIdx.x, tid = threadIdx.x;
    const float* row = proj + (size_t)t * ld;
    const int pos = positions[t];
    const int dq = d + rot, dk = rank + rot, half = rot_dims / 2;
    const float2* tab = half <= LAT_ANGLES ? angles : nullptr;
    if (tab) {
        for (int j = tid; j < half; j += blockDim.x) angles[j] = latent_angle(pos, inv_freq[j], mag);
        __syncthreads();
    }
    // queries: the plain part as it is, the rotated part turned by the position
    const int tf = short_row ? short_row[t] : t;                  // the token's row of q_plain and q_full
    if (tf < 0) {
        q_plain = nullptr;
        q_full = nullptr;
    } else if (short_row) {
        q_all = nullptr;
    }
    const auto rotate_one = [&](int e) {
        const int hh = e / rot, i = e % rot;
        const float* qr = row + hh * dq + d;
        const float v = latent_rotated(qr, i, half, halves, pos, inv_freq, mag, tab);
        if (q_full) q_full[((size_t)tf * H + hh) * dk + rank + i] = v;
        if (q_all) q_all[((size_t)t * H + hh) * dq + d + i] = from_f32<A>(v);
    };
    const bool vec = ((d | rot | ld) & 3) == 0 && (((size_t)proj | (size_t)q_plain | (size_t)q_all | (size_t)q_full) & 15) == 0;      // (rows of A: 4 elements)
    if (vec) {
        // a warp a head at a time, four elements a lane and four heads' loads under way; the turned parts as well where the
        // rotation turns all of them.  Bound by memory: 2,048 tokens of 16 heads of 128 + 64 (45 MB) took 20.8 us when a turned
        // element went by itself and every four elements divided for their head, now 13.7.
        const int lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5, groups = rot >> 2;
        const bool turn = rot_dims == rot && (halves ? half % 4 == 0 : 1) && tab && (!q_full || ((rank | dk) & 3) == 0);
        for (int i = lane * 4; i < d; i += 128)
            for (int h0 = warp; h0 < H; h0 += 4 * nw) {
                float4 v[4];
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    if (h0 + k * nw < H) v[k] = *reinterpret_cast<const float4*>(row + (h0 + k * nw) * dq + i);
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const int hh = h0 + k * nw;
                    if (hh >= H) break;
                    if (q_plain) store4<A>(q_plain + ((size_t)tf * H + hh) * d + i, v[k]);
                    if (q_all) store4<A>(q_all + ((size_t)t * H + hh) * dq + i, v[k]);
                }
            }
        if (turn) {
            for (int u = tid; u < H * groups; u += blockDim.x) {
                const int hh = u / groups, i = (u - hh * groups) * 4;
                const float* x = row + hh * dq + d;
                const float4 v = *reinterpret_cast<const float4*>(x + i);
                float4 y;
                if (halves) {
                    const int j = i < half ? i : i - half;
                    const float4 o = *reinterpret_cast<const float4*>(x + (i < half ? i + half : j));
                    const float2 a0 = tab[j], a1 = tab[j + 1], a2 = tab[j + 2], a3 = tab[j + 3];
                    y = i < half ? make_float4(v.x * a0.x - o.x * a0.y, v.y * a1.x - o.y * a1.y, v.z * a2.x - o.z * a2.y, v.w * a3.x - o.w * a3.y)
                                 : make_float4(v.x * a0.x + o.x * a0.y, v.y * a1.x + o.y * a1.y, v.z * a2.x + o.z * a2.y, v.w * a3.x + o.w * a3.y);
                } else {
                    const float2 a0 = tab[i >> 1], a1 = tab[(i >> 1) + 1];
                    y = make_float4(v.x * a0.x - v.y * a0.y, v.y * a0.x + v.x * a0.y, v.z * a1.x - v.w * a1.y, v.w * a1.x + v.z * a1.y);
                }
                if (q_full) store4<float>(q_full + ((size_t)tf * H + hh) * dk + rank + i, y);
                if (q_all) store4<A>(q_all + ((size_t)t * H + hh) * dq + d + i, y);
            }
        } else {
            for (int e = tid; e < H * rot; e += blockDim.x) rotate_one(e);
        }
    } else {
        for (int e = tid; e < H * d; e += blockDim.x) {
            const int hh = e / d, i = e % d;
            const A v = from_f32<A>(row[hh * dq + i]);
            if (q_plain) q_plain[((size_t)tf * H + hh) * d + i] = v;
            if (q_all) q_all[((size_t)t * H + hh) * dq + i] = v;
        }
        for (int e = tid; e < H * rot; e += blockDim.x) rotate_one(e);
    }
    if (!has_kv) return;
    const float* z = kv ? kv + (size_t)t * ld_kv : row + H * dq;
    float ss = 0.f;
    if (tid < LAT_PREP)                                 // always the same threads: a latent's bits do not depend on the step
        for (int i = tid; i < rank; i += LAT_PREP) ss += z[i] * z[i];
    ss = block_sum(ss, red);
    const float rinv = 1.0f / sqrtf(ss / (float)rank + eps);
    const int pidx = pos / P;
    const int page = (pos >= 0 && pidx < bt_width) ? block_table[(size_t)token_req[t] * bt_width + pidx] : -1;
    if (page < 0 || page >= num_pages) {
        if (tid == 0) atomicOr(err, AIE_DEV_PAGE_OOB);
        return;
    }
    C* dst = pages + ((size_t)page * P + (pos - pidx * P)) * dk;
    for (int i = tid; i < rank; i += blockDim.x) dst[i] = from_f32<C>((z[i] * rinv) * c_weight[i]);
    const float* kr = z + rank;
    for (int i = tid; i < rot; i += blockDim.x) dst[rank + i] = from_f32<C>(latent_rotated(kr, i, half, halves, pos, inv_freq, mag, tab));
}

extern "C" int aie_latent_prepare(const float* proj, int ld, int T, int H, int d, int rot, int rank, int rot_dims,
                                  int has_kv, const float* c_weight, float eps, const float* inv_freq, void* q_plain,
                                  int q_dtype, float* q_full, void* pages, int cache_dtype, const int* positions,
                                  const int* token_req, const int* block_table, int bt_width, int num_pages, int P,
                                  unsigned* err, const float* kv, int ld_kv, int halves, float mag, void* q_all,
                                  const int* short_row, cudaStream_t st) {
    if (T <= 0) return 0;
    if (rot_dims % 2 || rot_dims > rot || H <= 0 || d < 0 || rank <= 0) return AIE_BAD_ARG;
    const int threads = T <= 2 * aie_sm_count() ? 1024 : LAT_PREP;      // few tokens: a block has an SM to itself
#define GO(A, C)                                                                                                      \
    launch_pdl(latent_prepare_kernel<A, C>, dim3(T), dim3(threads), 0, st, proj, ld, H, d, rot, rank, rot_dims, has_kv, c_weight, eps, inv_freq, \
                                                   (A*)q_plain, q_full, (C*)pages, positions, token_req, block_table,  \
                                                   bt_width, num_pages, P, err, kv, ld_kv, halves, mag, (A*)q_all, short_row)
    if (q_dtype == AIE_F32 && cache_dtype == AIE_F32) GO(float, float);
    else if (q_dtype == AIE_BF16 && cache_dtype == AIE_BF16) GO(bf16, bf16);
    else if (q_dtype == AIE_BF16 && cache_dtype == AIE_F32) GO(bf16, float);
    else if (q_dtype == AIE_F32 && cache_dtype == AIE_BF16) GO(float, bf16);
    else return AIE_BAD_ARG;
#undef GO
    AIE_LAUNCH_CHECK();
}

// q_full [T, H, dk] float32 (folded plain part | rotated part); pages [num_pages, P, dk]; out [T, H, rank].
template <typename C, typename O, int NACC>
__global__ void __launch_bounds__(LAT_CHUNK)
latent_attention_kernel(const float* __restrict__ q_full, const C* __restrict__ pages, O* __restrict__ out,
                        const int* __restrict__ positions, const int* __restrict__ token_req,
                        const int* __restrict__ block_table, int bt_width, int num_pages, int P, int H, int rank,
                        int dk, int window, float scale, const float* __restrict__ sink, const int* __restrict__ q_len, unsigned* err) {
    extern __shared__ __align__(16) float sm[];
    float* q_s = sm;                                   // dk (rounded up to even)
    float* p_s = q_s + ((dk + 1) & ~1);                // CHUNK
    float* red = p_s + LAT_CHUNK;                      // 32
    long long* off_s = (long long*)(red + 32);         // CHUNK

    const int t = blockIdx.x, h = blockIdx.y, tid = threadIdx.x;
    const int pos = positions[t], row = token_req[t];
    if (q_len && q_len[row] == 1) return;              // lone tokens are another kernel's
    for (int e = tid; e < dk; e += blockDim.x) q_s[e] = q_full[((size_t)t * H + h) * dk + e];
    __syncthreads();

    int lo = 0;
    if (window > 0 && pos - window + 1 > 0) lo = pos - window + 1;
    float m = sink ? sink[h] : -INFINITY, l = sink ? 1.f : 0.f;      // the sink opens the running softmax
    float acc[NACC];
#pragma unroll
    for (int a = 0; a < NACC; ++a) acc[a] = 0.f;

    for (int c0 = (lo / LAT_CHUNK) * LAT_CHUNK; c0 <= pos; c0 += LAT_CHUNK) {
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
                off = ((long long)page * P + (kp % P)) * dk;
                const C* kr = pages + off;
                float dot = 0.f;
                for (int e = 0; e < dk; ++e) dot = fmaf(q_s[e], to_f32<C>(kr[e]), dot);
                s = dot * scale;
            }
        }
        off_s[tid] = off;
        const float cmax = block_max(s, red);
        const float m_new = fmaxf(m, cmax);
        const float p = (off >= 0) ? expf(s - m_new) : 0.f;
        const float corr = (m == -INFINITY) ? 0.f : expf(m - m_new);
        p_s[tid] = p;
        const float csum = block_sum(p, red);
        l = l * corr + csum;
        m = m_new;
#pragma unroll
        for (int a = 0; a < NACC; ++a) acc[a] *= corr;
        const int n = min(LAT_CHUNK, pos - c0 + 1);
        for (int j = 0; j < n; ++j) {
            const long long o = off_s[j];
            if (o < 0) continue;
            const float pj = p_s[j];
#pragma unroll
            for (int a = 0; a < NACC; ++a)
                if (tid + a * LAT_CHUNK < rank) acc[a] = fmaf(pj, to_f32<C>(pages[o + tid + a * LAT_CHUNK]), acc[a]);
        }
        __syncthreads();
    }
    const float inv = l > 0.f ? 1.0f / l : 0.f;
    O* o = out + ((size_t)t * H + h) * rank;
#pragma unroll
    for (int a = 0; a < NACC; ++a)
        if (tid + a * LAT_CHUNK < rank) o[tid + a * LAT_CHUNK] = from_f32<O>(acc[a] * inv);
}

template <typename C, typename O>
static int latent_go(const float* q_full, const void* pages, void* out, const int* positions, const int* token_req,
                     const int* block_table, int bt_width, int num_pages, int P, int T, int H, int rank, int dk,
                     int window, float scale, const float* sink, const int* q_len, unsigned* err, cudaStream_t st) {
    const size_t smem = (size_t)(((dk + 1) & ~1) + LAT_CHUNK + 32) * sizeof(float) + LAT_CHUNK * sizeof(long long);
    dim3 grid(T, H);
#define GO(N)                                                                                                        \
    latent_attention_kernel<C, O, N><<<grid, LAT_CHUNK, smem, st>>>(q_full, (const C*)pages, (O*)out, positions,     \
                                                                    token_req, block_table, bt_width, num_pages, P, \
                                                                    H, rank, dk, window, scale, sink, q_len, err)
    if (rank <= LAT_CHUNK) GO(1);
    else if (rank <= 2 * LAT_CHUNK) GO(2);
    else if (rank <= 4 * LAT_CHUNK) GO(4);
    else GO(8);
#undef GO
    AIE_LAUNCH_CHECK();
}

// q_len [requests] (or null): tokens of requests that bring one are left alone.
extern "C" int aie_latent_attention(const float* q_full, const void* pages, int cache_dtype, void* out, int out_dtype,
                                    const int* positions, const int* token_req, const int* block_table, int bt_width,
                                    int num_pages, int P, int T, int H, int rank, int dk, int window, float scale,
                                    const float* sink, const int* q_len, unsigned* err, cudaStream_t st) {
    if (T <= 0) return 0;
    if (rank <= 0 || dk < rank || H <= 0 || H > 65535) return AIE_BAD_ARG;
    if (rank > 8 * LAT_CHUNK || dk > 8192) return AIE_UNSUPPORTED;
    if (cache_dtype == AIE_F32 && out_dtype == AIE_F32)
        return latent_go<float, float>(q_full, pages, out, positions, token_req, block_table, bt_width, num_pages, P, T, H, rank, dk, window, scale, sink, q_len, err, st);
    if (cache_dtype == AIE_BF16 && out_dtype == AIE_BF16)
        return latent_go<bf16, bf16>(q_full, pages, out, positions, token_req, block_table, bt_width, num_pages, P, T, H, rank, dk, window, scale, sink, q_len, err, st);
    if (cache_dtype == AIE_BF16 && out_dtype == AIE_F32)
        return latent_go<bf16, float>(q_full, pages, out, positions, token_req, block_table, bt_width, num_pages, P, T, H, rank, dk, window, scale, sink, q_len, err, st);
    return AIE_BAD_ARG;
}
