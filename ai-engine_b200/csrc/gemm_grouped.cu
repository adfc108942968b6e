// Products of rows grouped by expert, C[row] = W[expert of the row's tile] . X[row] with X in tiles of 64 rows of one expert each
// (bfloat16, float32 sums in tensor memory): the kernel for experts that have several tiles, whose weights are then read for all of
// them at once.  gemm_tc.cu's grouped form takes one or two tiles a block and is bound by what its operands cost between L2 and
// shared memory (32 KB for 256 cycles of products); here an item is 128 rows of an expert's weights against up to four of its
// tiles (48 KB for 512 cycles), one block an SM (or two of a cluster) walks items, and an item's epilogue runs while the next one's products do:
//   warp 0 (one lane)  TMA loads of W [128 x 64] and of the tiles' X [64 x 64] into a ring of stages;
//   warp 1 (one lane)  four tcgen05.mma (K = 16) a stage into one of two accumulators of 256 columns;
//   warps 2-9          the epilogue of the accumulator before (lane = weight row, column = token; two warps share a quarter of the
//                      rows and take half of the columns each: with one the unit of a short K took longer than the products).
// Items are walked in steps of the grid, those of four tiles first, the weight tiles of the same X side by side.
// From a K of 1,024 on (and an even number of weight tiles) two blocks of a cluster share an item of 256 weight rows, with
// cta_group::2: each loads its own 128 rows and half of X's (32 KB a stage and SM instead of 48, so six stages), the first one issues
// the products of both, each block keeps the sums of its weight rows and has its own epilogue.  A short K is bound by the epilogue and
// loses what the pair costs to join (see gg_go).
// GLU: W [2 F, K] holds F gate rows, then F up rows.  A weight tile takes 64 of either in groups of 16, so that a warp's 32 lanes hold
// a unit's gate and up sixteen lanes apart; act = min(gate, limit) * sigmoid(slope * it) * (up kept within +-limit + shift), as
// clamped_glu makes it out of float32 sums, is stored in bfloat16.
// Bound by L2 (12 TB/s over the chip).  32 experts of 2,048 x 2,048, us, a launch by itself on a cold L2: 214 rows each 101 as two tiles a
// block, 85 as items of one block, 80 as items of two, 1,024 rows each 276, 231, 199; gate and up with the unit 120 (two kernels), 92, 89
// and 347, 237, 237.  An L2 policy that evicts the weights first: 72 -> 81.
// Every wait is bounded (see tc_common.cuh).
#include "tc_common.cuh"

#define GG_BM 128
#define GG_BK 64
#define GG_TILE 64          // rows of X a tile
#define GG_MOST 4           // tiles an item
#define GG_THREADS 320
#define GG_MAX_TILES 2048   // tiles of a launch
#define GG_W_BYTES (GG_BM * GG_BK * 2)
#define GG_X_BYTES (GG_TILE * GG_BK * 2)
#define GG_LIST_BYTES (GG_MAX_TILES * 8)
// CTAS: blocks that share an item (1 or 2)
template <int CTAS> struct GgSmem {
    static constexpr int x_bytes = GG_X_BYTES / CTAS, stage = GG_W_BYTES + GG_MOST * x_bytes, STAGES = CTAS == 2 ? 6 : 4;
    // [alignment slack | 1 KB: barriers | list of items | ring]
    static constexpr int bytes = 2048 + GG_LIST_BYTES + STAGES * stage;
};

struct GgGlu {
    float limit, slope, shift;
};

__device__ __forceinline__ unsigned gg_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;\n" : "=r"(r));
    return r;
}
__device__ __forceinline__ void gg_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n" ::: "memory");
    asm volatile("barrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}
__device__ __forceinline__ unsigned gg_first(unsigned long long* bar) {      // the cluster's first block's barrier
    unsigned at;
    asm volatile("mapa.shared::cluster.u32 %0, %1, 0;\n" : "=r"(at) : "r"(tc_smem(bar)));
    return at;
}
// a tile into this block's shared memory whose bytes count on the first block's barrier
__device__ __forceinline__ void gg_load_pair(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%3, %4}], [%2];\n"
                 ::"r"(tc_smem(dst)), "l"(map), "r"(gg_first(bar)), "r"(x), "r"(y) : "memory");
}
template <int CTAS>
__device__ __forceinline__ void gg_load(void* dst, const CUtensorMap* map, unsigned long long* bar, int x, int y) {
    if (CTAS == 2) gg_load_pair(dst, map, bar, x, y);
    else tma_load_2d(dst, map, bar, x, y);
}
template <int CTAS>
__device__ __forceinline__ void gg_mma(unsigned d, unsigned long long a, unsigned long long b, unsigned idesc, unsigned accumulate) {
    if (CTAS == 2)
        asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
                     "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}\n"
                     ::"r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
    else
        umma(d, a, b, idesc, accumulate);
}
template <int CTAS>
__device__ __forceinline__ void gg_commit(unsigned long long* bar) {      // ... on both blocks' barriers
    if (CTAS == 2)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;\n"
                     ::"r"(tc_smem(bar)), "h"((unsigned short)3) : "memory");
    else
        umma_commit(bar);
}
template <int CTAS>
__device__ __forceinline__ void gg_arrive_first(unsigned long long* bar) {      // on the first block's barrier
    if (CTAS == 2) {
        asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];\n" ::"r"(gg_first(bar)) : "memory");
    } else {
        mbar_arrive_plain(bar);
    }
}

template <bool GLU, int CTAS, typename OT>
__global__ void __launch_bounds__(GG_THREADS, 1)
gemm_grouped_kernel(const __grid_constant__ CUtensorMap map_w, const __grid_constant__ CUtensorMap map_x, OT* __restrict__ C,
                    const int* __restrict__ tile_w, int n_tiles, int N, int K, int ldc, unsigned* err, const GgGlu glu) {
    constexpr int STAGES = GgSmem<CTAS>::STAGES, STAGE = GgSmem<CTAS>::stage, XB = GgSmem<CTAS>::x_bytes;
    extern __shared__ unsigned char gg_raw[];
    unsigned char* bars = reinterpret_cast<unsigned char*>(((size_t)gg_raw + 1023) & ~(size_t)1023);
    unsigned long long* full = reinterpret_cast<unsigned long long*>(bars);
    unsigned long long* empty = full + STAGES;
    unsigned long long* acc_full = empty + STAGES;      // [2]
    unsigned long long* acc_empty = acc_full + 2;          // [2] the epilogue has read it
    unsigned* tmem_slot = reinterpret_cast<unsigned*>(acc_empty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    int* n_groups_s = reinterpret_cast<int*>(tmem_slot + 2);
    int* asked_s = n_groups_s + 1;                         // stages of the ring that this block asked for (see tc_drain)
    int2* list = reinterpret_cast<int2*>(bars + 1024);     // (first tile * 4 + tiles - 1, expert)
    unsigned char* ring = bars + 1024 + GG_LIST_BYTES;
    int* tw = reinterpret_cast<int*>(ring);                // the tiles' experts and the items that begin there, until the list is made
    unsigned char* code = ring + GG_MAX_TILES * 4;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        tma_prefetch_map(&map_w);
        tma_prefetch_map(&map_x);
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(&acc_full[a], 1);
            mbar_init(&acc_empty[a], 8 * CTAS);
        }
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
    }
    if (warp == 1) {
        if (CTAS == 2) {
            asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(tmem_slot)), "r"(512));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::);
        } else {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc_smem(tmem_slot)), "r"(512));
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::);
        }
    }
    pdl_launch_dependents();
    pdl_wait();                                            // the list of tiles and the rows are earlier kernels' output
    for (int i = tid; i < n_tiles; i += GG_THREADS) tw[i] = tile_w[i];
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const unsigned tmem = *tmem_slot;
    if (warp == 0) {
        // a run of an expert's tiles is cut into items of four from its start; the same list in every block
        int run = 0;
        for (int base = 0; base < n_tiles; base += 32) {
            const int y = base + lane;
            const int e = y < n_tiles ? tw[y] : -1;
            const unsigned starts = __ballot_sync(0xffffffffu, y == 0 || (y < n_tiles && tw[y - 1] != e));
            const unsigned mine = starts & (0xffffffffu >> (31 - lane));
            const int first = mine ? base + 31 - __clz(mine) : run;
            if (starts) run = base + 31 - __clz(starts);
            if (y < n_tiles) {
                int n = 0;
                if (e >= 0 && (y - first) % GG_MOST == 0) {
                    n = 1;
                    while (n < GG_MOST && y + n < n_tiles && tw[y + n] == e) ++n;
                }
                code[y] = (unsigned char)n;
            }
        }
        __syncwarp();
        int at = 0;
        for (int n = GG_MOST; n > 0; --n)
            for (int base = 0; base < n_tiles; base += 32) {
                const int y = base + lane;
                const bool takes = y < n_tiles && code[y] == n;
                const unsigned hit = __ballot_sync(0xffffffffu, takes);
                if (takes) list[at + __popc(hit & ((1u << lane) - 1))] = make_int2(y * 4 + n - 1, tw[y]);
                at += __popc(hit);
            }
        if (lane == 0) *n_groups_s = at;
    }
    asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");      // the ring was written to by threads
    if (CTAS == 2) gg_cluster_sync();                      // both blocks' barriers are there
    else __syncthreads();
    // an item: CTAS neighbouring weight tiles, one a block, against a group's rows, of which a block loads its part
    const int rank = CTAS == 2 ? (int)gg_rank() : 0, first_item = blockIdx.x / CTAS, step = gridDim.x / CTAS;
    const int per_tile = GLU ? GG_BM / 2 : GG_BM, NT = (GLU ? N / 2 : N) / per_tile / CTAS, items = *n_groups_s * NT;
    const int kbs = (K + GG_BK - 1) / GG_BK;

    if (warp == 0) {
        if (tc_elect()) {
            int s = 0, asked = 0;
            unsigned ph = 1;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += step) {
                const int2 g = list[item / NT];
                const int y = g.x >> 2, n = (g.x & 3) + 1, w0 = g.y * N + ((item % NT) * CTAS + rank) * per_tile;
                const int x0 = y * GG_TILE + rank * n * (GG_TILE / CTAS);
                for (int kb = 0; kb < kbs; ++kb) {
                    ok = mbar_wait(&empty[s], ph, abort_flag, err);
                    if (!ok) break;
                    unsigned char* st = ring + s * STAGE;
                    if (rank == 0) mbar_expect_tx(&full[s], CTAS * (GG_W_BYTES + n * XB));
                    if (GLU) {
#pragma unroll
                        for (int q = 0; q < 4; ++q) {
                            gg_load<CTAS>(st + q * 4096, &map_w, &full[s], kb * GG_BK, w0 + q * 16);
                            gg_load<CTAS>(st + q * 4096 + 2048, &map_w, &full[s], kb * GG_BK, w0 + N / 2 + q * 16);
                        }
                    } else {
                        gg_load<CTAS>(st, &map_w, &full[s], kb * GG_BK, w0);
                    }
                    for (int i = 0; i < n; ++i)
                        gg_load<CTAS>(st + GG_W_BYTES + i * XB, &map_x, &full[s], kb * GG_BK, x0 + i * (GG_TILE / CTAS));
                    ++asked;
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
            }
            *asked_s = asked;
            // a pair's products free the stages in both blocks: all have been freed before either block leaves
            for (int i = 0; CTAS == 2 && i < STAGES && ok; ++i) {
                ok = mbar_wait(&empty[s], ph, abort_flag, err);
                if (++s == STAGES) {
                    s = 0;
                    ph ^= 1;
                }
            }
        }
    } else if (warp == 1) {
        if (rank == 0 && tc_elect()) {
            int s = 0, a = 0;
            unsigned ph = 0, aph = 1;
            bool ok = true;
            for (int item = first_item; item < items && ok; item += step) {
                const int n = (list[item / NT].x & 3) + 1;
                const unsigned idesc = umma_idesc(n * GG_TILE) + (CTAS == 2 ? (128u >> 4) << 24 : 0u), d = tmem + (unsigned)(a * 256);
                ok = mbar_wait(&acc_empty[a], aph, abort_flag, err);
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                for (int kb = 0; kb < kbs; ++kb) {
                    ok = mbar_wait(&full[s], ph, abort_flag, err);
                    if (!ok) break;
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    unsigned char* st = ring + s * STAGE;
                    const unsigned long long da = umma_desc(st), db = umma_desc(st + GG_W_BYTES);
#pragma unroll
                    for (int j = 0; j < GG_BK / 16; ++j) gg_mma<CTAS>(d, da + 2 * j, db + 2 * j, idesc, (kb > 0 || j > 0) ? 1u : 0u);
                    gg_commit<CTAS>(&empty[s]);
                    if (++s == STAGES) {
                        s = 0;
                        ph ^= 1;
                    }
                }
                if (ok) gg_commit<CTAS>(&acc_full[a]);
                if (a == 1) aph ^= 1;
                a ^= 1;
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int a = 0;
        unsigned aph = 0;
        for (int item = first_item; item < items; item += step) {
            const int2 g = list[item / NT];
            const int n = (g.x & 3) + 1, t0 = (g.x >> 2) * GG_TILE, col0 = ((item % NT) * CTAS + rank) * per_tile;
            bool ok = true;
            if (lane == 0) ok = mbar_wait(&acc_full[a], aph, abort_flag, err);
            ok = __shfl_sync(0xffffffffu, ok ? 1 : 0, 0) != 0;
            if (!ok) break;
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
            const unsigned at = tmem + (unsigned)(a * 256) + ((unsigned)(quarter * 32) << 16);
#pragma unroll 1
            for (int c0 = half * 32 * n; c0 < (half + 1) * 32 * n; c0 += 32) {
                unsigned v[32];
                asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                             "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];\n"
                             : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
                               "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]),
                               "=r"(v[16]), "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]),
                               "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
                             : "r"(at + (unsigned)c0));
                asm volatile("tcgen05.wait::ld.sync.aligned;\n" ::: "memory");
                if (GLU) {
                    // lanes 0 .. 15 hold gates and take the even tokens, the others ups and the odd ones
                    const bool low = lane < 16;
                    OT* to = C + (size_t)(t0 + c0 + (low ? 0 : 1)) * ldc + col0 + quarter * 16 + (lane & 15);
#pragma unroll
                    for (int j = 0; j < 32; j += 2) {
                        const float own0 = __uint_as_float(v[j]), own1 = __uint_as_float(v[j + 1]);
                        const float other = __shfl_xor_sync(0xffffffffu, low ? own1 : own0, 16);
                        const float gate = fminf(low ? own0 : other, glu.limit);
                        const float up = fminf(fmaxf(low ? other : own1, -glu.limit), glu.limit);
                        to[(size_t)j * ldc] = from_f32<OT>(gate / (1.0f + expf(-glu.slope * gate)) * (up + glu.shift));
                    }
                } else {
                    OT* to = C + (size_t)(t0 + c0) * ldc + col0 + quarter * 32 + lane;
#pragma unroll
                    for (int j = 0; j < 32; ++j) to[(size_t)j * ldc] = from_f32<OT>(__uint_as_float(v[j]));
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            __syncwarp();
            if (lane == 0) gg_arrive_first<CTAS>(&acc_empty[a]);
            if (a == 1) aph ^= 1;
            a ^= 1;
        }
    }

    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    // a pair's copies all count on the first block's barriers, and both leave together: the second waits on one that nothing arrives
    // at until it runs out, which gives copies that the first had not armed yet their time
    if (*abort_flag && tid == 0) tc_drain(full, rank == 0 ? STAGES : 1, rank == 0 ? *asked_s : 1);
    __syncthreads();
    if (CTAS == 2) gg_cluster_sync();                      // nobody leaves while the other still reaches for its barriers
    if (warp == 1) {
        __syncwarp();
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (CTAS == 2) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
        else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
    }
}

template <bool GLU, int CTAS, typename OT>
static int gg_launch(const CUtensorMap& mw, const CUtensorMap& mx, void* C, const int* tile_w, int n_tiles, int N, int K, int ldc,
                     unsigned* err, const GgGlu& glu, cudaStream_t st) {
    auto kern = gemm_grouped_kernel<GLU, CTAS, OT>;
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, GgSmem<CTAS>::bytes);
    if (e != cudaSuccess) return (int)e;
    const long long most = (long long)n_tiles * (N / GG_BM), sms = aie_sm_count() / CTAS * CTAS;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)(most < sms ? most : sms));      // (a multiple of CTAS: N / 128 is)
    cfg.blockDim = dim3(GG_THREADS);
    cfg.dynamicSmemBytes = GgSmem<CTAS>::bytes;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[0].val.programmaticStreamSerializationAllowed = pdl_enabled() ? 1 : 0;
    attr[1].id = cudaLaunchAttributeClusterDimension;
    attr[1].val.clusterDim.x = CTAS;
    attr[1].val.clusterDim.y = attr[1].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = CTAS == 2 ? 2 : 1;
    e = cudaLaunchKernelEx(&cfg, kern, mw, mx, (OT*)C, tile_w, n_tiles, N, K, ldc, err, glu);
    return (int)e;
}

template <bool GLU, typename OT>
static int gg_go(const void* X, const void* W, void* C, const int* tile_w, int n_tiles, int N, int K, int ldc, int E, unsigned* err,
                 const GgGlu& glu, cudaStream_t st) {
    // Where two blocks take over, us as one block / as two (32 experts, N = 2,048, a launch by itself on a cold L2), at K = 512, 640, 768,
    // 896, 1,024, 1,536, 2,048: float32 results with 214 rows each 36/38 41/42 45/44 49/47 53/51 70/65 85/80, with 1,024 rows 99/96 109/101
    // 120/108 131/115 142/124 186/158 231/199; the unit with 214 rows 41/44 44/46 47/49 51/53 55/57 75/74 92/89, with 1,024 rows 115/122
    // 119/127 125/132 132/138 141/148 190/192 237/237.  Plain results gain from 768 on, the unit from some 1,500: one line between them.
    const int ctas = N / GG_BM % 2 || K < 1024 ? 1 : 2;
    CUtensorMap mw, mx;
    int rc = tc_make_map_2d(&mw, W, (unsigned long long)E * N, K, (unsigned long long)K * 2, GLU ? 16 : GG_BM, GG_BK);
    if (rc) return rc;
    rc = tc_make_map_2d(&mx, X, (unsigned long long)n_tiles * GG_TILE, K, (unsigned long long)K * 2, GG_TILE / ctas, GG_BK);
    if (rc) return rc;
    return ctas == 2 ? gg_launch<GLU, 2, OT>(mw, mx, C, tile_w, n_tiles, N, K, ldc, err, glu, st)
                     : gg_launch<GLU, 1, OT>(mw, mx, C, tile_w, n_tiles, N, K, ldc, err, glu, st);
}

// X [tiles * 64, K], W [E, N, K] bfloat16, tile_w [tiles] (-1: the tile is skipped and its rows of C are left as they are).  C [rows, ldc]
// float32 or bfloat16; with `glu` (W holds N / 2 gate rows, then as many up rows) C [rows, ldc >= N / 2] is bfloat16.
extern "C" int aie_gemm_grouped(const void* X, const void* W, void* C, int out_dtype, int tiles, int N, int K, int ldc, int E,
                                const int* tile_w, int glu, float limit, float slope, float shift, unsigned* err, cudaStream_t stream) {
    if (tiles <= 0 || N <= 0) return 0;
    if (!tile_w || E <= 0) return AIE_BAD_ARG;
    if (K <= 0 || K % 8 || N % GG_BM || tiles > GG_MAX_TILES || ((size_t)X & 15) || ((size_t)W & 15) ||
        (long long)E * N > 0x7fffffffLL || (glu && out_dtype != AIE_BF16))
        return AIE_UNSUPPORTED;
    const GgGlu g{limit, slope, shift};
#define GO(GLU, OT) return gg_go<GLU, OT>(X, W, C, tile_w, tiles, N, K, ldc, E, err, g, stream)
    if (glu) GO(true, bf16);
    if (out_dtype == AIE_F32) GO(false, float);
    if (out_dtype == AIE_BF16) GO(false, bf16);
#undef GO
    return AIE_BAD_ARG;
}
