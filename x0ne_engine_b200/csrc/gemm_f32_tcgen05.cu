// C[M,N] = A[M,K] * W[N,K]^T of float32 operands on the tensor cores, no less precise than float32 multiply-adds.
//
// Every operand value x is cut into two TF32 values, hi = x rounded to 11 significant bits and lo = x - hi (of which the unit
// takes 11 bits again: together 22 to 24 bits of x), and a product is hi hi + hi lo + lo hi; the dropped lo lo is below 2^-24 of it.
// The products themselves are exact; what the tensor core loses is in its sums, which it cuts off instead of rounding.  So the
// accumulator in tensor memory only ever holds ONE slab of 32 values of k (the small terms first, then four steps of the large ones),
// and float32 registers add the slabs with rounding:  slab sums along a part of K, K in eight parts, the parts in order.  That order
// is a property of K alone: it is the same whatever M is, wherever the output lies, and however the parts are spread over blocks, so
// a row's result is bit-identical alone, in a batch, in a prompt or in a decode step.
//
// What bounds it: shared memory.  A slab of a 128 x 128 tile keeps the tensor core busy for 768 cycles (12 products of 128 x 128 x 8), and moves 16 KB
// of W and of x in, out to the splitting warps, 32 KB of split x in and 48 KB out to the tensor core: 1,150 cycles of shared memory; the slabs
// take about 1,550.  W's split operand goes to tensor memory for that reason.  Few rows: a product of 128 x 16 x 8 takes the tensor core as long as
// one of 128 x 128 x 8 (63 cycles), 768 a slab again, in which a multiprocessor streams 21 bytes of W a cycle.
// Against gemm_f32.cu's kernels, us: 8 / 64 / 200 / 600 rows of 2048 x 2048 19.8 / 65 / 142 / 260 -> 10.0 / 14.5 / 29 / 49, of 12288 x 2048 48 / 231 / 479 / 1069
// -> 27 / 42 / 95 / 233, of 2048 x 6144 55 / 190 / 424 / 768 -> 21 / 31 / 62 / 128.
//
// Results that are not finite, or not zero and below 2^-60, are computed again as one chain of multiply-adds (gemm_f32.cu's
// arithmetic): infinities and NaN have no split, values near the end of the float32 range no room for their low half.
#include "tcgen05.cuh"

#define SP_K 32                 // values of k per slab: a 128-byte row of shared memory
#define SP_PARTS 8              // K's parts
#define SP_TILE_W 128           // rows of W per block: the tensor memory's lanes

template <int NX> struct SpConfig {
    static constexpr int A_BYTES = SP_TILE_W * 128, X_BYTES = NX * 128;
    static constexpr int RAW = NX >= 96 ? 3 : 4;                     // stages of operands as they come
    static constexpr int ACC = NX >= 96 ? 3 : 4;                     // accumulators
    static constexpr int SPLIT = NX == 128 || NX == 32 ? 2 : NX == 64 ? 4 : 3;       // stages of split operands (W: tensor memory, x: shared memory)
    static constexpr int TMEM = NX <= 32 ? 256 : 512;                // columns: two accumulators, then 64 per split stage
    static constexpr int A_COL = ACC * NX;
    static constexpr int BLOCKS = NX <= 32 ? 2 : 1;
    // Warps that split x.  Where registers run out (the adding warps hold up to 128 sums a thread), warpgroups trade them: 640 threads start
    // with 96 each, the adding 256 take GROW and the other 384 keep SHRINK (256 GROW + 384 SHRINK <= 640 x 96).
    // The pool may be just as large as what is asked for, so nobody takes registers back before the adding warps are through with
    // theirs: a barrier of all warps (of the cluster, or of the block alone) stands between every warp's first trade and its second, and behind it
    // the adding warps give back without waiting for anything.
    static constexpr int X_WARP = NX >= 64 ? 16 : 14, X_WARPS = NX >= 64 ? 4 : 2, THREADS = 32 * (X_WARP + X_WARPS);
    static constexpr int START = 96, GROW = NX >= 96 ? 168 : 136, SHRINK = NX >= 96 ? 48 : 64;
    static constexpr bool SHIFT_REGS = NX >= 64;
    static_assert(!SHIFT_REGS || (THREADS == 640 && 256 * GROW + 384 * SHRINK <= 640 * START && 640 * START <= 65536), "registers");
    static constexpr int TILES = RAW * (A_BYTES + X_BYTES) + SPLIT * 2 * X_BYTES;
    static_assert(ACC >= SPLIT, "a split stage is free when its slab's accumulator is full, which must not become full again before the stage is waited for");
    static_assert(A_COL + 64 * SPLIT <= TMEM, "tensor memory");
};

struct SpShared {
    uint64_t raw_full[8], raw_empty[8], split_full[4], acc_full[4], acc_empty[4];
    uint32_t tmem_base;
    int failed;
};

struct SpArgs {
    const float* A;
    const float* W;
    float* C;
    int M, N, K, xt, tma, w_batched, x_batched;
    int64_t lda, ldw, ldc, sa, sw, sc;
    int* status;
};

// TF32 products: A from tensor memory (a column per value of k), B from shared memory
__device__ __forceinline__ void sp_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::tf32 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void sp_st16(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
                 "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]) : "memory");
}
__device__ __forceinline__ void sp_ld8(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}
__device__ __forceinline__ void sp_ld16(uint32_t taddr, uint32_t* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]) : "r"(taddr) : "memory");
}
// x rounded to TF32 (ties away from zero), and what is left of x cut off to TF32
__device__ __forceinline__ uint32_t sp_hi(float x) { return (__float_as_uint(x) + 0x1000u) & 0xffffe000u; }
__device__ __forceinline__ uint32_t sp_lo(float x, uint32_t hi) { return __float_as_uint(x - __uint_as_float(hi)) & 0xffffe000u; }

// One output as a chain of multiply-adds over k = 0, 1, ...
__device__ __noinline__ float sp_chain(const float* a, const float* w, int K) {
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(a[k], w[k], acc);
    return acc;
}
__device__ __forceinline__ bool sp_irregular(float v) {
    const uint32_t e = __float_as_uint(v) & 0x7fffffffu;
    return e >= 0x7f800000u || e - 1u < ((127u - 60u) << 23) - 1u;
}

// All warps of the block, from either side of the split into roles.
template <int THREADS> __device__ __forceinline__ void sp_all_warps() { asm volatile("bar.sync 1, %0;" ::"n"(THREADS) : "memory"); }

// NX: rows of x per block.  CL: blocks of a cluster, each with 8 / CL parts of K.
//
// Warps 0-7 add the slabs (warp & 3: the quarter of the lanes they may read, warp >> 2: the half of the columns).  Warps 8-11 split
// W into tensor memory, the last ones x into shared memory; warp 12 brings both in, warp 13 issues the products.
template <int NX, int CL>
__global__ void __launch_bounds__(SpConfig<NX>::THREADS, SpConfig<NX>::BLOCKS) gemm_f32_split_kernel(const __grid_constant__ CUtensorMap map_x, const __grid_constant__ CUtensorMap map_w,
                                                                                           SpArgs a) {
    using Cfg = SpConfig<NX>;
    constexpr int COLS = NX / 2, OWN = SP_PARTS / CL, RAW = Cfg::RAW, SPLIT = Cfg::SPLIT;
    constexpr int LD = COLS % 16 == 0 ? 16 : 8;
    extern __shared__ unsigned char sp_dyn[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sp_dyn) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw_w = base;                                        // [stage][128 rows][128 bytes], 128-byte swizzle
    unsigned char* raw_x = raw_w + RAW * Cfg::A_BYTES;                  // [stage][NX rows][128 bytes]
    unsigned char* split_x = raw_x + RAW * Cfg::X_BYTES;                // [stage][hi, lo][NX rows][128 bytes]
    SpShared* sh = reinterpret_cast<SpShared*>(base + Cfg::TILES);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0), lane = threadIdx.x & 31;
    const int rank = CL > 1 ? (int)(blockIdx.x % CL) : 0, tile = blockIdx.x / CL;
    const int m0 = tile % a.xt * NX, n0 = tile / a.xt * SP_TILE_W, z = blockIdx.z;
    const int slabs = (a.K + SP_K - 1) / SP_K, part = (slabs + SP_PARTS - 1) / SP_PARTS;
    const int first = min(slabs, rank * OWN * part), last = min(slabs, (rank + 1) * OWN * part);      // this block's slabs

    if (threadIdx.x == 0) {
        for (int s = 0; s < RAW; ++s) {
            mbar_init(&sh->raw_full[s], a.tma ? 1 : 32);
            mbar_init(&sh->raw_empty[s], 4 + Cfg::X_WARPS);
        }
        for (int s = 0; s < SPLIT; ++s) {
            mbar_init(&sh->split_full[s], 4 + Cfg::X_WARPS);
        }
        for (int b = 0; b < Cfg::ACC; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            mbar_init(&sh->acc_empty[b], 8);
        }
        sh->failed = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (warp == 12 && lane == 0 && a.tma) {
        tma_prefetch_map(&map_w);
        tma_prefetch_map(&map_x);
    }
    if (warp == 13) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc_smem(&sh->tmem_base)), "r"(Cfg::TMEM) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    pdl_launch_dependents();
    tc_fence_after();
    const uint32_t tmem = sh->tmem_base;
    bool ok = true;
    auto passed = [&](uint64_t* bar, int parity, int code) { return mbar_try_wait(bar, parity) || mbar_wait(bar, parity, a.status, code); };
    auto wait = [&](uint64_t* bar, int parity, int code) {
        if (ok) ok = __all_sync(0xffffffffu, passed(bar, parity, code));
    };
    // where a role stands in a ring of n stages: the stage, and the parity of this round's phase
    struct Ring {
        int at = 0, round = 0;
        __device__ __forceinline__ void next(int n) {
            if (++at == n) {
                at = 0;
                round ^= 1;
            }
        }
    };
    float* xch = reinterpret_cast<float*>(base);            // [part][NX][128 / CL]: the parts of this block's share of the outputs
    constexpr int SHARE = SP_TILE_W / CL;

    if (warp < 8) {
        if constexpr (Cfg::SHIFT_REGS) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::GROW));
        const int quarter = warp & 3, half = warp >> 2;
        const uint32_t trow = tmem + ((uint32_t)(quarter * 32) << 16) + half * COLS;
        constexpr int KEEP = CL > 1 ? OWN : 2;              // parts in registers: a block's own, or the sum so far and the next one
        float sum[KEEP][COLS];
#pragma unroll
        for (int p = 0; p < KEEP; ++p)
#pragma unroll
            for (int c = 0; c < COLS; ++c) sum[p][c] = 0.f;
        Ring acc;
        auto add_part = [&](float (&to)[COLS], int n) {
            for (int i = 0; i < n; ++i, acc.next(Cfg::ACC)) {
                const int b = acc.at;
                wait(&sh->acc_full[b], acc.round, 20);
                tc_fence_after();
                uint32_t r[COLS <= 32 ? COLS : 32];
#pragma unroll
                for (int c0 = 0; c0 < COLS; c0 += 32) {
                    constexpr int STEP = COLS < 32 ? COLS : 32;
#pragma unroll
                    for (int c = 0; c < STEP && c0 + c < COLS; c += LD) {
                        if constexpr (LD == 16) sp_ld16(trow + b * NX + c0 + c, r + c);
                        else sp_ld8(trow + b * NX + c0 + c, r + c);
                    }
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (c0 + 32 >= COLS) {
                        tc_fence_before();
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh->acc_empty[b]);
                    }
#pragma unroll
                    for (int c = 0; c < STEP && c0 + c < COLS; ++c) to[c0 + c] += __uint_as_float(r[c]);
                }
            }
        };
        pdl_wait();
        if constexpr (CL > 1) {
#pragma unroll
            for (int p = 0; p < OWN; ++p) add_part(sum[p], max(0, min(slabs, (rank * OWN + p + 1) * part) - min(slabs, (rank * OWN + p) * part)));
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");        // every block of the cluster is done with its tiles
            // the outputs of lanes r SHARE .. go to block r, part by part
            const int l = quarter * 32 + lane, owner = l / SHARE;
            uint32_t to;
            asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(to) : "r"(tc_smem(xch)), "r"(owner));
#pragma unroll
            for (int p = 0; p < OWN; ++p)
#pragma unroll
                for (int c = 0; c < COLS; ++c)
                    asm volatile("st.shared::cluster.f32 [%0], %1;" ::"r"(to + 4u * (uint32_t)(((rank * OWN + p) * NX + half * COLS + c) * SHARE + l % SHARE)), "f"(sum[p][c]) : "memory");
            // (back to the launch's registers for what all warps run)
            if constexpr (Cfg::SHIFT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::START));
        } else {
            add_part(sum[0], min(slabs, part));
            for (int p = 1; p < SP_PARTS; ++p) {
                add_part(sum[1], max(0, min(slabs, (p + 1) * part) - min(slabs, p * part)));
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    sum[0][c] += sum[1][c];
                    sum[1][c] = 0.f;
                }
            }
            const int n = n0 + quarter * 32 + lane;
            if (n < a.N && ok) {
                const float* w = a.W + (int64_t)z * a.sw + (int64_t)n * a.ldw;
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    const int m = m0 + half * COLS + c;
                    if (m < a.M) {
                        float v = sum[0][c];
                        if (sp_irregular(v)) v = sp_chain(a.A + (int64_t)z * a.sa + (int64_t)m * a.lda, w, a.K);
                        a.C[(int64_t)z * a.sc + (int64_t)m * a.ldc + n] = v;
                    }
                }
            }
            __syncwarp();
            if constexpr (Cfg::SHIFT_REGS) {
                sp_all_warps<Cfg::THREADS>();
                asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::START));
            }
        }
    } else {
        if constexpr (Cfg::SHIFT_REGS) asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Cfg::SHRINK));
        if (warp < 12) {
            const int row = (warp & 3) * 32 + lane;
            const uint32_t tlane = tmem + ((uint32_t)((warp & 3) * 32) << 16) + Cfg::A_COL;
            Ring raw, split, acc;
            for (int it = 0; it < last - first; ++it, raw.next(RAW), split.next(SPLIT)) {
                wait(&sh->raw_full[raw.at], raw.round, 21);
                if (!ok) break;
                const unsigned char* src = raw_w + raw.at * Cfg::A_BYTES + row * 128;
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    float x[16];
                    uint32_t hi[16];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 v = *reinterpret_cast<const float4*>(src + (((4 * g + c) ^ (row & 7)) << 4));
                        x[4 * c] = v.x; x[4 * c + 1] = v.y; x[4 * c + 2] = v.z; x[4 * c + 3] = v.w;
                    }
#pragma unroll
                    for (int e = 0; e < 16; ++e) {
                        hi[e] = sp_hi(x[e]);
                        x[e] = __uint_as_float(sp_lo(x[e], hi[e]));
                    }
                    if (g == 1) {
                        __syncwarp();
                        if (lane == 0) mbar_arrive(&sh->raw_empty[raw.at]);
                    } else if (it >= SPLIT) {          // (a split stage is free when its slab's accumulator is full)
                        wait(&sh->acc_full[acc.at], acc.round, 22);
                        acc.next(Cfg::ACC);
                        tc_fence_after();
                    }
                    if (ok) {
                        sp_st16(tlane + split.at * 64 + 16 * g, hi);
                        sp_st16(tlane + split.at * 64 + 32 + 16 * g, reinterpret_cast<const uint32_t*>(x));
                    }
                }
                if (!ok) break;
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->split_full[split.at]);
            }
        } else if (warp >= Cfg::X_WARP) {
            constexpr int XT = 32 * Cfg::X_WARPS;
            const int t = threadIdx.x - Cfg::X_WARP * 32;
            constexpr int PIECES = NX * 8 / XT, BATCH = PIECES < 8 ? PIECES : PIECES % 8 == 0 ? 8 : PIECES / 2;      // 16-byte pieces of a slab per thread, and at a time
            static_assert(PIECES % BATCH == 0, "pieces");
            Ring raw, split, acc;
            for (int it = 0; it < last - first; ++it, raw.next(RAW), split.next(SPLIT)) {
                wait(&sh->raw_full[raw.at], raw.round, 23);
                const float4* src = reinterpret_cast<const float4*>(raw_x + raw.at * Cfg::X_BYTES) + t;       // (the split tiles keep its swizzle)
                uint4* dst = reinterpret_cast<uint4*>(split_x + split.at * 2 * Cfg::X_BYTES) + t;
#pragma unroll
                for (int i0 = 0; i0 < PIECES; i0 += BATCH) {
                    float4 v[BATCH];
                    if (ok)
#pragma unroll
                        for (int i = 0; i < BATCH; ++i) v[i] = src[XT * (i0 + i)];
                    if (i0 == 0 && it >= SPLIT) {
                        wait(&sh->acc_full[acc.at], acc.round, 24);
                        acc.next(Cfg::ACC);
                    }
                    if (!ok) break;
#pragma unroll
                    for (int i = 0; i < BATCH; ++i) {
                        const uint4 h = make_uint4(sp_hi(v[i].x), sp_hi(v[i].y), sp_hi(v[i].z), sp_hi(v[i].w));
                        dst[XT * (i0 + i)] = h;
                        dst[NX * 8 + XT * (i0 + i)] = make_uint4(sp_lo(v[i].x, h.x), sp_lo(v[i].y, h.y), sp_lo(v[i].z, h.z), sp_lo(v[i].w, h.w));
                    }
                }
                if (!ok) break;
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sh->raw_empty[raw.at]);
                    mbar_arrive(&sh->split_full[split.at]);
                }
            }
        } else if (warp == 12) {
            pdl_wait();             // (W may be a product's result too)
            asm volatile("fence.proxy.async.global;" ::: "memory");
            int issued = 0;
            Ring raw;
            for (int it = 0; it < last - first; ++it, raw.next(RAW)) {
                const int rs = raw.at, k0 = (first + it) * SP_K;
                if (it >= RAW) wait(&sh->raw_empty[rs], raw.round ^ 1, 25);
                if (!ok) break;
                if (a.tma) {
                    if (lane == 0) {
                        mbar_expect_tx(&sh->raw_full[rs], Cfg::A_BYTES + Cfg::X_BYTES);
                        tma_load_3d(raw_w + rs * Cfg::A_BYTES, &map_w, k0, n0, a.w_batched ? z : 0, &sh->raw_full[rs]);
                        tma_load_3d(raw_x + rs * Cfg::X_BYTES, &map_x, k0, m0, a.x_batched ? z : 0, &sh->raw_full[rs]);
                    }
                    __syncwarp();
                } else {            // rows that TMA cannot address: value by value, a lane per k
                    const int k = k0 + lane;
                    auto rows = [&](unsigned char* dst, const float* from, int64_t ld, int r0, int n, int end) {
                        for (int r = 0; r < n; ++r) {
                            const bool in = r0 + r < end && k < a.K;
                            const uint32_t d = tc_smem(dst + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4);
                            const float* s = in ? from + (int64_t)(r0 + r) * ld + k : from;
                            const int bytes = in ? 4 : 0;
                            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(d), "l"(s), "r"(bytes) : "memory");
                        }
                    };
                    rows(raw_w + rs * Cfg::A_BYTES, a.W + (int64_t)z * a.sw, a.ldw, n0, SP_TILE_W, a.N);
                    rows(raw_x + rs * Cfg::X_BYTES, a.A + (int64_t)z * a.sa, a.lda, m0, NX, a.M);
                    asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(tc_smem(&sh->raw_full[rs])) : "memory");
                }
                ++issued;
            }
            if (!ok) {              // copies that nobody waited for must land before the block's memory is given back
                if (!a.tma) asm volatile("cp.async.wait_all;" ::: "memory");
                else
                    for (int it = max(0, issued - RAW); it < issued; ++it) mbar_wait(&sh->raw_full[it % RAW], (it / RAW) & 1, a.status, 21);
            }
        } else if (warp == 13) {
            // instruction descriptor: f32 accumulate, TF32 operands, both K-major, M = 128, N = NX
            constexpr uint32_t idesc = (1u << 4) | (2u << 7) | (2u << 10) | ((uint32_t)(NX >> 3) << 17) | ((128u >> 4) << 24);
            // One thread issues; the next slab's waits come ahead of a slab's last products, so that the unit's queue does not run dry.
            uint32_t leader = 0;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leader));
            if (leader) {
                Ring acc, split, acc_now, split_now;         // of the slab that is waited for, and of the one that is issued
                auto ready = [&](int it) {
                    if (it >= last - first) return;
                    if (it >= Cfg::ACC) ok = ok && passed(&sh->acc_empty[acc.at], acc.round ^ 1, 26);
                    ok = ok && passed(&sh->split_full[split.at], split.round, 27);
                    acc.next(Cfg::ACC);
                    split.next(SPLIT);
                };
                ready(0);
                for (int it = 0; it < last - first && ok; ++it, acc_now.next(Cfg::ACC), split_now.next(SPLIT)) {
                    const int ss = split_now.at, b = acc_now.at;
                    tc_fence_after();
                    const uint32_t d = tmem + b * NX, wa = tmem + Cfg::A_COL + ss * 64, xh = tc_smem(split_x + ss * 2 * Cfg::X_BYTES), xl = xh + Cfg::X_BYTES;
#pragma unroll
                    for (int k = 0; k < 4; ++k) sp_mma(d, wa + 32 + 8 * k, tc_desc(xh + 32 * k), idesc, k > 0 ? 1u : 0u);
#pragma unroll
                    for (int k = 0; k < 4; ++k) sp_mma(d, wa + 8 * k, tc_desc(xl + 32 * k), idesc, 1u);
                    ready(it + 1);
#pragma unroll
                    for (int k = 0; k < 4; ++k) sp_mma(d, wa + 8 * k, tc_desc(xh + 32 * k), idesc, 1u);
                    tc_commit(&sh->acc_full[b]);
                }
            }
            __syncwarp();
        }
        if (CL > 1) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
        }
        __syncwarp();
        if constexpr (Cfg::SHIFT_REGS) {
            if (CL == 1) sp_all_warps<Cfg::THREADS>();
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Cfg::START));
        }
    }
    if constexpr (CL > 1) {
        __syncwarp();
        asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");            // every part of this block's share has arrived
        if (warp >= 8) pdl_wait();
        for (int i = threadIdx.x; i < SHARE * NX; i += Cfg::THREADS) {
            const int l = i % SHARE, c = i / SHARE, m = m0 + c, n = n0 + rank * SHARE + l;
            float v = xch[c * SHARE + l];
#pragma unroll
            for (int p = 1; p < SP_PARTS; ++p) v += xch[(p * NX + c) * SHARE + l];
            if (m < a.M && n < a.N) {
                if (sp_irregular(v)) v = sp_chain(a.A + (int64_t)z * a.sa + (int64_t)m * a.lda, a.W + (int64_t)z * a.sw + (int64_t)n * a.ldw, a.K);
                a.C[(int64_t)z * a.sc + (int64_t)m * a.ldc + n] = v;
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 13) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(Cfg::TMEM) : "memory");
    }
}

// ----------------------------------------------------------------------------------------
// host
// ----------------------------------------------------------------------------------------
template <int NX, int CL>
static int sp_launch(SpArgs a, int batch, cudaStream_t stream) {
    using Cfg = SpConfig<NX>;
    static_assert(CL == 1 || SP_PARTS / CL * NX / 2 <= 64, "parts in registers");
    static_assert(SP_PARTS * NX * (SP_TILE_W / CL) * 4 <= Cfg::TILES || CL == 1, "exchange");
    CUtensorMap mx = {}, mw = {};
    if (a.tma) {
        if (int e = x0ne_tc_make_map_3d_f32(&mx, a.A, a.K, a.M, a.x_batched ? batch : 1, a.lda, a.x_batched ? a.sa : a.lda * a.M, NX)) return e;
        if (int e = x0ne_tc_make_map_3d_f32(&mw, a.W, a.K, a.N, a.w_batched ? batch : 1, a.ldw, a.w_batched ? a.sw : a.ldw * a.N, SP_TILE_W)) return e;
    }
    const size_t smem = Cfg::TILES + sizeof(SpShared) + 1024;
    static OncePerDevice configured;
    if (configured.need()) {
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_split_kernel<NX, CL>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        X0NE_REQUIRE(e == cudaSuccess, "gemm_f32: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured.done();
    }
    a.xt = (a.M + NX - 1) / NX;
    const int64_t blocks = (int64_t)a.xt * ((a.N + SP_TILE_W - 1) / SP_TILE_W) * CL;
    X0NE_REQUIRE(blocks <= 0x7fffffff, "gemm_f32: too many tiles");
    if (CL > 1) x0ne_launch_clusters(gemm_f32_split_kernel<NX, CL>, dim3((unsigned)blocks, 1, batch), dim3(Cfg::THREADS), CL, smem, stream, mx, mw, a);
    else x0ne_launch(gemm_f32_split_kernel<NX, CL>, dim3((unsigned)blocks, 1, batch), dim3(Cfg::THREADS), smem, stream, mx, mw, a);
    X0NE_LAUNCH_CHECK();
}

// Which form a product takes.  All give the same bits, so only time decides: what each takes, in us, from its tiles per multiprocessor
// and the slabs a block walks.  Measured at K 2,048 and 6,144 and one tile per multiprocessor, a slab being 128 x NX x 32:
//   rows of x       16     32     64     96    128
//   per slab       0.43   0.52   0.53   0.59   0.81    (16 and 32: two blocks fit a multiprocessor, and take 0.37 and 0.41 each when they share it;
//                                                     0.60 and 0.70 where many such blocks stream W from memory)
//   start, end      2.9    2.7    4.6    8.5    8.2    one block walks K;  3 to 5.5 in a cluster
// so 96 rows of x per tile are the cheapest per output, fewer where they leave padding, and a cluster pays where tiles leave
// multiprocessors idle.  (Clusters of 8, and of 2 or 4 blocks that may share a multiprocessor, do not reach all of them: 16 clusters of 8 one to
// a multiprocessor take two rounds, 14 take one.)  Against all forms at 8 to 2,048 rows and 20 sizes of W its choice is the fastest or within
// 10 % of it at all but a few.
struct SpForm {
    int nx, cl;
    float slab, shared, ends;
};
static const SpForm SP_FORMS[] = {
    {16, 1, 0.60f, 0.37f, 2.9f}, {16, 2, 0.43f, 0.37f, 3.5f}, {16, 4, 0.43f, 0.37f, 3.1f}, {16, 8, 0.43f, 0.37f, 3.3f}, {32, 1, 0.70f, 0.41f, 2.7f},
    {32, 4, 0.52f, 0.41f, 4.0f}, {32, 8, 0.52f, 0.41f, 3.7f}, {64, 1, 0.53f, 0.f, 4.6f}, {64, 4, 0.53f, 0.f, 5.0f}, {64, 8, 0.53f, 0.f, 4.3f},
    {96, 1, 0.59f, 0.f, 8.5f}, {128, 1, 0.81f, 0.f, 8.2f}, {128, 8, 0.81f, 0.f, 5.5f},
};
static int sp_choose(int64_t M, int64_t N, int64_t K, int64_t batch, int64_t sms) {
    const int64_t slabs = (K + SP_K - 1) / SP_K, part = (slabs + SP_PARTS - 1) / SP_PARTS;
    double best = 0;
    int form = 0;
    for (const SpForm& f : SP_FORMS) {
        if (f.nx / 2 >= (M > 9 ? M : 9)) continue;          // half of its rows would be padding
        const int64_t tiles = (M + f.nx - 1) / f.nx * ((N + SP_TILE_W - 1) / SP_TILE_W) * batch * f.cl;
        if (tiles > 0x7fffffff) continue;
        const int64_t reached = f.cl == 1 || (f.nx == 64 && f.cl == 4) || sms < 4 ? sms : sms * 3 / 4;
        const double turns = (double)((tiles + reached - 1) / reached), walk = (double)(f.cl == 1 ? slabs : part * (SP_PARTS / f.cl));
        const double us = f.shared > 0.f ? (turns > 2 ? turns / 2 : 1) * f.ends + walk * (turns > 1 ? turns * f.shared : f.slab) : turns * (f.ends + walk * f.slab);
        if (form == 0 || us < best) {
            best = us;
            form = f.nx * 16 + f.cl;
        }
    }
    return form;
}

// The product on the tensor cores.  `status`: one int in device memory, zero before the first call; bits 20 to 27 say that a wait ran out.
// `form`: 0 by size, else NX * 16 + CL (measurements and tests).
X0NE_API int x0ne_gemm_f32_split(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, int batch, int64_t sa, int64_t sw,
                                 int64_t sc, int form, int* status, cudaStream_t stream) {
    X0NE_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N && status != nullptr, "gemm_f32: M %d N %d K %d", M, N, K);
    X0NE_REQUIRE(batch >= 1 && batch <= 65535, "gemm_f32: batch %d", batch);
    if (M == 0) return 0;
    SpArgs a = {A, W, C, M, N, K, 0, 0, batch > 1 && sw != 0, batch > 1 && sa != 0, lda, ldw, ldc, sa, sw, sc, status};
    a.tma = lda % 4 == 0 && ldw % 4 == 0 && sa % 4 == 0 && sw % 4 == 0 && sa >= 0 && sw >= 0 && ((((uintptr_t)A) | ((uintptr_t)W)) & 15) == 0;
    switch (form != 0 ? form : sp_choose(M, N, K, batch, x0ne_sm_count())) {
        case 16 * 16 + 1: return sp_launch<16, 1>(a, batch, stream);
        case 16 * 16 + 2: return sp_launch<16, 2>(a, batch, stream);
        case 16 * 16 + 4: return sp_launch<16, 4>(a, batch, stream);
        case 16 * 16 + 8: return sp_launch<16, 8>(a, batch, stream);
        case 32 * 16 + 1: return sp_launch<32, 1>(a, batch, stream);
        case 32 * 16 + 4: return sp_launch<32, 4>(a, batch, stream);
        case 32 * 16 + 8: return sp_launch<32, 8>(a, batch, stream);
        case 64 * 16 + 1: return sp_launch<64, 1>(a, batch, stream);
        case 64 * 16 + 4: return sp_launch<64, 4>(a, batch, stream);
        case 64 * 16 + 8: return sp_launch<64, 8>(a, batch, stream);
        case 96 * 16 + 1: return sp_launch<96, 1>(a, batch, stream);
        case 128 * 16 + 1: return sp_launch<128, 1>(a, batch, stream);
        case 128 * 16 + 8: return sp_launch<128, 8>(a, batch, stream);
    }
    X0NE_REQUIRE(false, "gemm_f32: no form %d for M %d N %d", form, M, N);
}
