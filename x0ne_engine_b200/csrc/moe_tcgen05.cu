// The experts' products of a routed feed-forward on the 5th-generation tensor cores, for passes with
// many (row, choice) pairs: the pairs of one expert lie together (moe.cu lists them), so a 128-row tile
// of one expert's pairs times a 256-row tile of that expert's weight is one tcgen05 accumulator, and
// the whole layer is one launch over a table of tiles that the grouping kernel wrote on the device.
//
//   up:   A = the rows gathered into the listed order [places][K] (moe_gather_rows), W = up weights
//         [experts x N][K]; the epilogue writes relu(.)^2 as bfloat16 to act[place][N]
//   down: A = act [places][K], W = down weights [experts x N][K]; the epilogue writes float32 to
//         y[pair][N], the pair looked up from the list (a row of the tile is one thread's)
//   gated up: W = [experts x N][K] with N = 2 x the experts' inner width, an expert's rows in blocks of 256: 128 gate
//         rows, then the 128 up rows of the same outputs; a tile's accumulator then holds a gate value and its up value
//         128 columns apart, and the epilogue writes silu(gate) * up as bfloat16 to act[place][N / 2]
//
// The pipeline is the one of gemm_tcgen05.cu: a copy thread (TMA, 128-byte swizzle, 4 stages), an MMA
// thread (accumulator double-buffered in tensor memory) and eight epilogue warps; blocks are
// persistent over the tiles.  How many tiles are real is read from device memory (the launch is sized
// for the worst case), so the launch depends on the host only through sizes.  A tile's A rows past the
// expert's last pair and W rows past the expert's last output row are read (the next expert's, or
// zeros past the end) and their results dropped.  Every barrier wait is bounded; a wait that runs out
// sets its bit in `status`, and the kernel frees its tensor memory and returns.
//
// The down product's float32 rows go out through shared memory in pieces of 64 bytes, four lanes each: written by the thread that holds the
// row, 16 bytes at a time, they were what bounded it (8,192 pairs of 1,024 -> 2,048: 52 us, 32 without any stores, 41 now; 32,000 pairs 198, 107, 157).
#include "tcgen05.cuh"

#define MT_BM 128
#define MT_BN 256
#define MT_BK 64
#define MT_STAGES 4
#define MT_EPILOGUE_WARPS 8             // two per quarter of a tile's rows, half of the columns each
#define MT_THREADS (64 + 32 * MT_EPILOGUE_WARPS)
#define MT_PITCH 20                     // floats between the rows of a warp's staged piece: 32 rows x 16 columns
#define MT_TMEM_COLS 512

struct MtShared {
    uint64_t full[MT_STAGES];
    uint64_t empty[MT_STAGES];
    uint64_t accum_full[2];
    uint64_t accum_empty[2];
    uint32_t tmem_base;
    int failed;
    __align__(16) float piece[MT_EPILOGUE_WARPS][32 * MT_PITCH];
};

#define MT_UP 0
#define MT_DOWN 1
#define MT_GATED 2

// What a warp does with its 32 rows of an accumulator (from column `trow` on): this thread's row of the tile goes to `row` of the results (< 0:
// nowhere).  It takes the `part`-th of `parts` shares of the columns.
template <int MODE>
__device__ __forceinline__ void mt_results(uint32_t trow, void* out, int N, int n0, int64_t row, int part, int parts, float* piece, int lane) {
    if (MODE == MT_GATED) {
        // columns c and 128 + c of the tile are the gate and the up value of output n0 / 2 + c (N is a multiple of 256)
        const int half = N / 2, chunks = MT_BN / 64 / parts;
#pragma unroll 1
        for (int c = part * chunks; c < (part + 1) * chunks; ++c) {
            float v[32], u[32];
            tc_ld32(trow + c * 32, v);
            tc_ld32(trow + MT_BN / 2 + c * 32, u);
            if (row < 0) continue;
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = v[i] / (1.0f + __expf(-v[i])) * u[i];
            bf16* dst = (bf16*)out + row * half + n0 / 2 + c * 32;
            if ((((uintptr_t)dst) & 15) == 0) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) tc_store8(dst + i, v + i);
            } else {
                for (int i = 0; i < 32; ++i) dst[i] = __float2bfloat16_rn(v[i]);
            }
        }
        return;
    }
    const int chunks = MT_BN / 32 / parts;
#pragma unroll 1
    for (int c = part * chunks; c < (part + 1) * chunks; ++c) {
        const int n = n0 + c * 32;
        if (n >= N) break;                          // (uniform over the warp)
        float v[32];
        tc_ld32(trow + c * 32, v);
        if (MODE == MT_DOWN && n + 32 <= N && N % 4 == 0 && (((uintptr_t)out) & 15) == 0) {
            // rows of 64 bytes, four lanes each: a thread's own row would go out in 16-byte pieces, 32 rows at a time
#pragma unroll
            for (int h = 0; h < 32; h += 16) {
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 16; i += 4) *reinterpret_cast<float4*>(piece + lane * MT_PITCH + i) = make_float4(v[h + i], v[h + i + 1], v[h + i + 2], v[h + i + 3]);
                __syncwarp();
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int r = 8 * i + (lane >> 2);
                    const int64_t to = __shfl_sync(0xffffffffu, row, r);
                    if (to >= 0) *reinterpret_cast<float4*>((float*)out + to * N + n + h + 4 * (lane & 3)) = *reinterpret_cast<const float4*>(piece + r * MT_PITCH + 4 * (lane & 3));
                }
            }
            continue;
        }
        if (row < 0) continue;
        if (MODE == MT_UP) {
#pragma unroll
            for (int i = 0; i < 32; ++i) {
                const float x = fmaxf(v[i], 0.f);
                v[i] = x * x;
            }
            bf16* dst = (bf16*)out + row * N + n;
            if (n + 32 <= N && (((uintptr_t)dst) & 15) == 0) {
#pragma unroll
                for (int i = 0; i < 32; i += 8) tc_store8(dst + i, v + i);
            } else {
                for (int i = 0; i < 32; ++i)
                    if (n + i < N) dst[i] = __float2bfloat16_rn(v[i]);
            }
        } else {
            float* dst = (float*)out + row * N + n;
            for (int i = 0; i < 32; ++i)
                if (n + i < N) dst[i] = v[i];
        }
    }
}

template <int MODE>
__global__ void __launch_bounds__(MT_THREADS) moe_tc_kernel(const __grid_constant__ CUtensorMap map_a,
                                                            const __grid_constant__ CUtensorMap map_w, void* __restrict__ out,
                                                            int N, int K, const int32_t* listed,
                                                            const int32_t* tiles, const int32_t* n_real_p,
                                                            int max_tiles, int n_tiles_n, int* status) {
    extern __shared__ unsigned char mt_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(mt_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int A_BYTES = MT_BM * 128, B_BYTES = MT_BN * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    MtShared* sh = reinterpret_cast<MtShared*>(base + MT_STAGES * STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k_blocks = (K + MT_BK - 1) / MT_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MT_STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->accum_full[b], 1);
            mbar_init(&sh->accum_empty[b], 32 * MT_EPILOGUE_WARPS);
        }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)),
                     "r"(MT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();          // the table of tiles, the list and the A rows were written by the kernels before this one
    // the A rows were written with ordinary stores and are read by TMA: order the two proxies on this side as well
    asm volatile("fence.proxy.async;" ::: "memory");
    int n_real = n_real_p[0];
    if (n_real > max_tiles) n_real = max_tiles;
    const int total = n_real * n_tiles_n;      // tile id -> (m tile = id % n_real, n tile = id / n_real)

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int tile = blockIdx.x; tile < total && !sh->failed; tile += gridDim.x) {
                const int mt = tile % n_real, n0 = (tile / n_real) * MT_BN;
                const int e = tiles[3 * mt], first = tiles[3 * mt + 1];
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % MT_STAGES;
                    if (it >= MT_STAGES && !mbar_wait(&sh->empty[s], ((it / MT_STAGES) - 1) & 1, status, 1)) {
                        sh->failed = 1;
                        break;
                    }
                    unsigned char* a = base + s * STAGE_BYTES;
                    mbar_expect_tx(&sh->full[s], STAGE_BYTES);
                    tma_load_2d(a, &map_a, kb * MT_BK, first, &sh->full[s]);
                    tma_load_2d(a + A_BYTES, &map_w, kb * MT_BK, e * N + n0, &sh->full[s]);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0) {
            // instruction descriptor: f32 accumulate, bf16 x bf16, both K-major, N = 256, M = 128
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((128u >> 4) << 24);
            int it = 0, t = 0;
            for (int tile = blockIdx.x; tile < total && !sh->failed; tile += gridDim.x, ++t) {
                const int ab = t & 1;
                const uint32_t acc_tmem = tmem + ab * 256;
                if (t >= 2 && !mbar_wait(&sh->accum_empty[ab], ((t >> 1) - 1) & 1, status, 4)) {
                    sh->failed = 1;
                    break;
                }
                tc_fence_after();
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % MT_STAGES;
                    if (!mbar_wait(&sh->full[s], (it / MT_STAGES) & 1, status, 2)) {
                        sh->failed = 1;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = tc_smem(base + s * STAGE_BYTES), b = a + A_BYTES;
#pragma unroll
                    for (int k = 0; k < MT_BK / 16; ++k)
                        tc_mma(acc_tmem, tc_desc(a + k * 32), tc_desc(b + k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit(&sh->empty[s]);
                }
                tc_commit(&sh->accum_full[ab]);
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int t = 0;
        for (int tile = blockIdx.x; tile < total; tile += gridDim.x, ++t) {
            const int ab = t & 1;
            const int mt = tile % n_real, n0 = (tile / n_real) * MT_BN;
            const int first = tiles[3 * mt + 1], count = tiles[3 * mt + 2];
            const int r = quarter * 32 + lane;
            int64_t row = -1;                              // the output row of this thread, or none
            if (r < count) row = MODE != MT_DOWN ? (int64_t)(first + r) : (int64_t)listed[first + r];
            if (!mbar_wait(&sh->accum_full[ab], (t >> 1) & 1, status, 3) || sh->failed) {
                sh->failed = 1;
                break;
            }
            tc_fence_after();
            mt_results<MODE>(tmem + ab * 256 + ((uint32_t)(quarter * 32) << 16), out, N, n0, row, half, 2, sh->piece[warp - 2], lane);
            tc_fence_before();
            mbar_arrive(&sh->accum_empty[ab]);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MT_TMEM_COLS) : "memory");
    }
}

// ----------------------------------------------------------------------------------------
// The same on pairs of blocks (cta_group::2, as gemm_tcgen05.cu's): a pair takes 256 listed pairs of one expert and 256 of its weight rows,
// each block 128 of both, and fetches 32 KB for every 512 cycles of products where a single block fetches 48.  A tile of 256 x 256 x 2,048 takes a pair
// 13 us, two of 128 x 256 x 2,048 take single blocks 16.5 (the clock falls under dense products, 13 us are 512 cycles per 64 of K at 1.26 GHz);
// which is ahead is a matter of rounds (`moe_tc_in_pairs` in ops.py).
// ----------------------------------------------------------------------------------------
#define MT2_STAGES 6
#define MT2_EPILOGUE_WARPS 8            // two per quarter of a block's rows, half of the columns each
#define MT2_THREADS (64 + 32 * MT2_EPILOGUE_WARPS)

struct Mt2Shared {
    uint64_t full[MT2_STAGES];
    uint64_t empty[MT2_STAGES];
    uint64_t accum_full[2];
    uint64_t accum_empty[2];
    uint32_t tmem_base;
    int failed;
    __align__(16) float piece[MT2_EPILOGUE_WARPS][32 * MT_PITCH];
};

template <int MODE>
__global__ void __launch_bounds__(MT2_THREADS) moe_tc_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_w, void* __restrict__ out, int N,
                                                                  int K, const int32_t* listed, const int32_t* tiles, const int32_t* n_real_p, int max_tiles, int n_tiles_n,
                                                                  int* status) {
    extern __shared__ unsigned char mt_raw[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(mt_raw) + 1023) & ~(uintptr_t)1023);
    constexpr int A_BYTES = 128 * 128, B_BYTES = 128 * 128, STAGE_BYTES = A_BYTES + B_BYTES;
    Mt2Shared* sh = reinterpret_cast<Mt2Shared*>(base + MT2_STAGES * STAGE_BYTES);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1, k_blocks = (K + MT_BK - 1) / MT_BK;

    if (threadIdx.x == 0) {
        for (int s = 0; s < MT2_STAGES; ++s) {
            mbar_init(&sh->full[s], 1);
            mbar_init(&sh->empty[s], 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(&sh->accum_full[b], 1);
            mbar_init(&sh->accum_empty[b], 2 * 32 * MT2_EPILOGUE_WARPS);     // the epilogue threads of both blocks
        }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(MT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pdl_launch_dependents();
    cluster_sync();          // both blocks' barriers are initialised before either block uses the other's
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    pdl_wait();              // the table of tiles, the list and the A rows were written by the kernels before this one
    asm volatile("fence.proxy.async;" ::: "memory");
    int n_real = n_real_p[0];
    if (n_real > max_tiles) n_real = max_tiles;
    const int total = n_real * n_tiles_n;      // tile id -> (m tile = id % n_real, n tile = id / n_real)

    if (warp == 0) {
        if (lane == 0) {
            int it = 0;
            for (int tile = pair; tile < total && !sh->failed; tile += pairs) {
                const int mt = tile % n_real, n0 = (tile / n_real) * MT_BN;
                const int e = tiles[3 * mt], first = tiles[3 * mt + 1] + 128 * (int)rank;
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % MT2_STAGES;
                    if (it >= MT2_STAGES && !mbar_wait(&sh->empty[s], ((it / MT2_STAGES) - 1) & 1, status, 1)) {
                        sh->failed = 1;
                        break;
                    }
                    unsigned char* a = base + s * STAGE_BYTES;
                    // the first block's barrier counts the bytes of both blocks
                    const uint32_t bar0 = cluster_addr(tc_smem(&sh->full[s]), 0);
                    if (rank == 0) mbar_expect_tx(&sh->full[s], 2 * STAGE_BYTES);
                    tma_load_2d_pair(a, &map_a, kb * MT_BK, first, bar0);
                    tma_load_2d_pair(a + A_BYTES, &map_w, kb * MT_BK, e * N + n0 + 128 * (int)rank, bar0);
                }
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && rank == 0) {
            // instruction descriptor: f32 accumulate, bf16 x bf16, both K-major, M = 256 over the pair, N = 256
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((256u >> 3) << 17) | ((256u >> 4) << 24);
            int it = 0, t = 0;
            for (int tile = pair; tile < total && !sh->failed; tile += pairs, ++t) {
                const int ab = t & 1;
                if (t >= 2 && !mbar_wait(&sh->accum_empty[ab], ((t >> 1) - 1) & 1, status, 4)) {
                    sh->failed = 1;
                    break;
                }
                tc_fence_after();
                for (int kb = 0; kb < k_blocks; ++kb, ++it) {
                    const int s = it % MT2_STAGES;
                    if (!mbar_wait(&sh->full[s], (it / MT2_STAGES) & 1, status, 2)) {
                        sh->failed = 1;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = tc_smem(base + s * STAGE_BYTES), b = a + A_BYTES;
#pragma unroll
                    for (int k = 0; k < MT_BK / 16; ++k)
                        tc_mma_pair(tmem + ab * 256, tc_desc(a + k * 32), tc_desc(b + k * 32), idesc, (kb > 0 || k > 0) ? 1u : 0u);
                    tc_commit_pair(&sh->empty[s]);
                }
                tc_commit_pair(&sh->accum_full[ab]);
            }
        }
    } else {
        const int quarter = warp & 3, half = (warp - 2) >> 2;
        int t = 0;
        for (int tile = pair; tile < total; tile += pairs, ++t) {
            const int ab = t & 1;
            const int mt = tile % n_real, n0 = (tile / n_real) * MT_BN;
            const int first = tiles[3 * mt + 1], count = tiles[3 * mt + 2];
            const int r = 128 * (int)rank + quarter * 32 + lane;
            int64_t row = -1;                              // the output row of this thread, or none
            if (r < count) row = MODE != MT_DOWN ? (int64_t)(first + r) : (int64_t)listed[first + r];
            if (!mbar_wait(&sh->accum_full[ab], (t >> 1) & 1, status, 3) || sh->failed) {
                sh->failed = 1;
                break;
            }
            tc_fence_after();
            mt_results<MODE>(tmem + ab * 256 + ((uint32_t)(quarter * 32) << 16), out, N, n0, row, half, 2, sh->piece[warp - 2], lane);
            tc_fence_before();
            mbar_arrive_cluster(cluster_addr(tc_smem(&sh->accum_empty[ab]), 0));
        }
    }
    tc_fence_before();
    __syncthreads();
    cluster_sync();          // neither block leaves while the other may still touch its memory or barriers
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(MT_TMEM_COLS) : "memory");
    }
}

// xs[place] = x[listed[place] / top] for the places that hold a pair (their number is offsets[experts]).
__global__ void moe_gather_rows_kernel(const bf16* x, int K, const int32_t* listed,
                                       const int32_t* offsets, int experts, int top, bf16* __restrict__ xs) {
    pdl_prologue();
    const int place = blockIdx.x;
    if (place >= offsets[experts]) return;
    const bf16* src = x + (int64_t)(listed[place] / top) * K;
    bf16* dst = xs + (int64_t)place * K;
    if (K % 8 == 0 && ((((uintptr_t)x | (uintptr_t)xs) & 15) == 0)) {
        for (int i = threadIdx.x * 8; i < K; i += blockDim.x * 8) *reinterpret_cast<uint4*>(dst + i) = *reinterpret_cast<const uint4*>(src + i);
    } else {
        for (int i = threadIdx.x; i < K; i += blockDim.x) dst[i] = src[i];
    }
}

template <int MODE>
static int moe_pair_launch(const CUtensorMap& map_a, const CUtensorMap& map_w, void* out, int N, int K, const int32_t* listed, const int32_t* tiles, const int32_t* n_real,
                           int max_tiles, int sms, int* status, cudaStream_t stream) {
    const size_t smem = (size_t)MT2_STAGES * (128 * 128 * 2) + sizeof(Mt2Shared) + 1024;
    static OncePerDevice configured;
    if (configured.need()) {
        const cudaError_t e = cudaFuncSetAttribute(moe_tc_pair_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        X0NE_REQUIRE(e == cudaSuccess, "moe_product_tc: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured.done();
    }
    const int n_tiles_n = (N + MT_BN - 1) / MT_BN;
    const int64_t worst = (int64_t)max_tiles * n_tiles_n, most = sms / 2 > 0 ? sms / 2 : 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(2 * (unsigned)(worst < most ? worst : most));
    cfg.blockDim = dim3(MT2_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 2;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaLaunchKernelEx(&cfg, moe_tc_pair_kernel<MODE>, map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, n_tiles_n, status);
    X0NE_LAUNCH_CHECK();
}

X0NE_API int x0ne_moe_gather_rows(const void* x, int K, const int32_t* listed, const int32_t* offsets, int experts, int top,
                                  void* xs, int pairs, cudaStream_t stream) {
    X0NE_REQUIRE(K > 0 && experts > 0 && top > 0 && pairs >= 0, "moe_gather: K %d experts %d top %d", K, experts, top);
    if (pairs == 0) return 0;
    x0ne_launch(moe_gather_rows_kernel, dim3(pairs), dim3(K >= 2048 ? 256 : 128), 0, stream, (const bf16*)x, K, listed, offsets, experts,
                top, (bf16*)xs);
    X0NE_LAUNCH_CHECK();
}

// which 0: up (a: gathered rows [a_rows][K], out: bfloat16 act [places][N]); which 1: down (a: act [a_rows][K], out:
// float32 y [pairs][N]); which 2: gated up (a as for 0, w rows in blocks of 128 gate and 128 up rows, N a multiple of 256,
// out: bfloat16 act [places][N / 2]).  w: [experts][N][K] bfloat16.  tiles: [max_tiles][3] from the grouping kernel run with
// tiles of 128 pairs (`pair` = 1, pairs of blocks: of 256); n_real: how many of them are real (device memory).
X0NE_API int x0ne_moe_product_tc(int which, const void* a, int64_t a_rows, const void* w, int experts, int N, int K,
                                 const int32_t* listed, const int32_t* tiles, const int32_t* n_real, int max_tiles, void* out,
                                 int pair, int* status, cudaStream_t stream) {
    X0NE_REQUIRE((which == 0 || which == 1 || which == 2) && experts > 0 && N > 0 && K > 0 && K % 8 == 0 && a_rows > 0 && max_tiles >= 0,
                 "moe_product_tc: experts %d N %d K %d (K must be a multiple of 8)", experts, N, K);
    X0NE_REQUIRE(which != 2 || N % MT_BN == 0, "moe_product_tc: gated experts of %d rows (blocks of %d)", N, MT_BN);
    X0NE_REQUIRE(status != nullptr && n_real != nullptr, "moe_product_tc: no status word or no tile count");
    X0NE_REQUIRE((((uintptr_t)a | (uintptr_t)w) & 15) == 0, "moe_product_tc: operands are not 16-byte aligned");
    if (max_tiles == 0) return 0;
    CUtensorMap map_a, map_w;
    if (int e = x0ne_tc_make_map(&map_a, a, a_rows, K, MT_BM)) return e;
    if (int e = x0ne_tc_make_map(&map_w, w, (int64_t)experts * N, K, pair ? 128 : MT_BN)) return e;
    if (pair) {
        const int sms = x0ne_sm_count();
        if (which == 0) return moe_pair_launch<MT_UP>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, sms, status, stream);
        if (which == 2) return moe_pair_launch<MT_GATED>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, sms, status, stream);
        return moe_pair_launch<MT_DOWN>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, sms, status, stream);
    }
    const size_t smem = (size_t)MT_STAGES * (MT_BM * 128 + MT_BN * 128) + sizeof(MtShared) + 1024;
    static OncePerDevice configured;
    if (configured.need()) {
        cudaError_t e1 = cudaFuncSetAttribute(moe_tc_kernel<MT_UP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaError_t e2 = cudaFuncSetAttribute(moe_tc_kernel<MT_DOWN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        cudaError_t e3 = cudaFuncSetAttribute(moe_tc_kernel<MT_GATED>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e1 != cudaSuccess || e2 != cudaSuccess || e3 != cudaSuccess) {
            x0ne_set_error("moe_product_tc: cannot set %zu bytes of shared memory", smem);
            return (int)(e1 != cudaSuccess ? e1 : (e2 != cudaSuccess ? e2 : e3));
        }
        configured.done();
    }
    const int n_tiles_n = (N + MT_BN - 1) / MT_BN;
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    if (sms <= 0) sms = 1;
    const int64_t worst = (int64_t)max_tiles * n_tiles_n;
    const int grid = worst < sms ? (int)worst : sms;
    // Launched without the early-start attribute: the kernel before it writes, with ordinary stores at its very end, the rows
    // this one reads by TMA a moment later.  Replayed from a graph with the early start, short prompt passes with many padding
    // rows gave other logits than the same launches made one by one (which leave more time between the two kernels); with a
    // plain launch and the proxy fence in the kernel they give the same bits.  The kernel still lets its own successor start early.
    if (which == 0)
        moe_tc_kernel<MT_UP><<<grid, MT_THREADS, smem, stream>>>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, n_tiles_n, status);
    else if (which == 2)
        moe_tc_kernel<MT_GATED><<<grid, MT_THREADS, smem, stream>>>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, n_tiles_n, status);
    else
        moe_tc_kernel<MT_DOWN><<<grid, MT_THREADS, smem, stream>>>(map_a, map_w, out, N, K, listed, tiles, n_real, max_tiles, n_tiles_n, status);
    X0NE_LAUNCH_CHECK();
}
