// Chunks of CT tokens of the step's portions, for kernels whose blocks each take one: requests in order, those that bring
// fewer than min_len tokens left out.
#pragma once
#include "common.cuh"

template <int CT> __device__ __forceinline__ int chunk_count(const int* q_len, int R, int min_len, int r) {
    const int n = r < R ? q_len[r] : 0;
    return n >= min_len ? (n + CT - 1) / CT : 0;
}

// Request r and chunk c of the idx-th of them; r < 0: there is none.  All threads of the block call it; found: two ints of
// shared memory.
template <int CT>
__device__ __forceinline__ void chunk_find(const int* q_len, int R, int min_len, int idx, int* found, int& r, int& c) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int rr = -1, cc = 0, before = 0;
        for (int base = 0; base < R && rr < 0; base += 32) {
            const int m = chunk_count<CT>(q_len, R, min_len, base + lane);
            int run = m;
            for (int o = 1; o < 32; o <<= 1) {
                const int up = __shfl_up_sync(0xffffffffu, run, o);
                if (lane >= o) run += up;
            }
            const unsigned hit = __ballot_sync(0xffffffffu, idx < before + run);
            if (hit) {
                const int l = __ffs(hit) - 1;
                rr = base + l;
                cc = idx - before - __shfl_sync(0xffffffffu, run - m, l);
            }
            before += __shfl_sync(0xffffffffu, run, 31);
        }
        if (lane == 0) {
            found[0] = rr;
            found[1] = cc;
        }
    }
    __syncthreads();
    r = found[0];
    c = found[1];
}

// Request r of the idx-th of those portions and the number of its first chunk; r < 0: there is none.  All threads of the block
// call it; found: two ints of shared memory.
template <int CT>
__device__ __forceinline__ void portion_find(const int* q_len, int R, int min_len, int idx, int* found, int& r, int& first) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int rr = -1, portions = 0, chunks = 0;
        for (int base = 0; base < R && rr < 0; base += 32) {
            int m = chunk_count<CT>(q_len, R, min_len, base + lane);
            unsigned takes = __ballot_sync(0xffffffffu, m > 0);
            const int n = __popc(takes);
            if (idx < portions + n) {
                for (int i = portions; i < idx; ++i) takes &= takes - 1;
                const int l = __ffs(takes) - 1;
                rr = base + l;
                if (lane >= l) m = 0;
            }
            portions += n;
            chunks += __reduce_add_sync(0xffffffffu, m);
        }
        if (lane == 0) {
            found[0] = rr;
            found[1] = chunks;
        }
    }
    __syncthreads();
    r = found[0];
    first = found[1];
}
