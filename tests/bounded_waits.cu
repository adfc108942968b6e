// Kernels of the tests of bounded waits: a ring whose last copies land late, or never.
#define TC_DRAIN_LIMIT (1u << 14)
#include "tc_common.cuh"

// `asked` copies of 16 bytes around a ring of `stages`; those of the last round come after `late` cycles (late < 0: never).  out[s]: the
// first word that stage s holds once tc_drain has returned (0: nothing came).
__global__ void late_copies_kernel(const int* __restrict__ src, int* __restrict__ out, int stages, int asked, long long late) {
    __shared__ __align__(16) int ring[8][4];
    __shared__ unsigned long long full[8];
    const int tid = threadIdx.x, before = max(asked - stages, 0);      // copies that land at once
    const auto copy = [&](int i) {
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], 16, [%2];\n"
                     ::"r"(tc_smem(ring[i % stages])), "l"(src + 4 * i), "r"(tc_smem(&full[i % stages])) : "memory");
    };
    if (tid == 0) {
        for (int s = 0; s < 8; ++s) {
            mbar_init(&full[s], 1);
            ring[s][0] = 0;
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
        for (int i = 0; i < asked; ++i) {
            mbar_expect_tx(&full[i % stages], 16);
            if (i >= before) continue;
            copy(i);
            for (unsigned k = 0; k < (1u << 20) && !mbar_try_wait(&full[i % stages], (i / stages) & 1); ++k) {}
        }
        for (int s = 0; s < stages; ++s) ring[s][0] = 0;
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    __syncthreads();
    if (tid == 32 && late >= 0) {
        const long long t0 = clock64();
        while (clock64() - t0 < late) {}
        for (int i = before; i < asked; ++i) copy(i);
    }
    if (tid == 0) {
        tc_drain(full, stages, asked);
        for (int s = 0; s < stages; ++s) out[s] = ring[s][0];
        for (int s = 0; s < stages && s < asked && late >= 0; ++s)      // (nothing is left in flight should the test fail)
            for (unsigned k = 0; k < (1u << 20) && !mbar_try_wait(&full[s], ((asked - 1 - s) / stages) & 1); ++k) {}
    }
    __syncthreads();
}

extern "C" int late_copies(const int* src, int* out, int stages, int asked, long long late, cudaStream_t st) {
    if (stages < 1 || stages > 8 || asked < 0 || asked > 64 || late > 1000000) return AIE_BAD_ARG;
    late_copies_kernel<<<1, 64, 0, st>>>(src, out, stages, asked, late);
    AIE_LAUNCH_CHECK();
}
