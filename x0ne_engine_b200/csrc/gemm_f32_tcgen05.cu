// C[M,N] = A[M,K] * W[N,K]^T of float32 operands on the tensor cores, no less precise than float32 multiply-adds.
//
// Every operand value x is cut into three bfloat16 values, x = a + b + c exactly (8 bits each of its 24, and the exponent range is float32's own),
// and a product is a a + (a b + b a) + (a c + b b + c a) + (b c + c b); the dropped c c is below 2^-32 of it.  The products of parts are exact; what
// the tensor core loses is in its sums, which it cuts off instead of rounding.  So the accumulator of the a a in tensor memory only ever holds ONE
// slab of 32 values of k, and float32 registers add the slabs with rounding; the small products, 2^-7 of the sum and less, have accumulators of
// their own by size, so that they lose nothing to the large ones, for a whole part of K.  Order: slab sums along a part of K, the part's small
// products, K in eight parts, the parts in order.  That order is a property of K alone: it is the same whatever M is, wherever the output lies, and
// however the parts are spread over blocks, so a row's result is bit-identical alone, in a batch, in a prompt or in a decode step.
// A product alone in its row, or beside zeros, is rounded once, as a multiply-add rounds it (2^-24 of it, and 2^-29 at most from its small parts);
// W the identity gives x back.
//
// What bounds it: a block's chain from slab to slab (operands in, split, products), in which no unit is busy all the time: 350 rows of
// 4096 x 2048 in tiles of 96 have the tensor core at work for 37 % of the cycles, shared memory for 47 %, issue slots for 45 %.  W's parts go to tensor memory,
// x's stand one behind the other in shared memory, so that one product takes a part of W against two or three of x.
// Against gemm_f32.cu's kernels, us (weights from memory): 8 / 64 / 200 / 600 rows of 2048 x 2048 20.0 / 63 / 147 / 254 -> 11.6 / 17.9 / 34.9 / 72.5, of
// 12288 x 2048 49 / 230 / 479 / 1076 -> 33.3 / 53.7 / 140 / 344, of 2048 x 6144 56 / 190 / 426 / 773 -> 24.7 / 38.9 / 76 / 190.  Three TF32 values took 1.05 to
// 1.1 times as long, two (23 bits of x) 0.7 to 0.9.
//
// Results that are not finite, or small beside what operands may have lost below the float32 range (`sp_irregular`), are computed again as one
// chain of multiply-adds (gemm_f32.cu's arithmetic): infinities and NaN have no split, values near the end of the range no room for their low parts.
#include "tcgen05.cuh"

#define SP_K 32                 // values of k per slab: a 128-byte row of shared memory
#define SP_PARTS 8              // K's parts
#define SP_TILE_W 128           // rows of W per block: the tensor memory's lanes

template <int NX> struct SpConfig {
    static constexpr int A_BYTES = SP_TILE_W * 128, X_BYTES = NX * 128;      // of a slab, as it comes
    static constexpr int RAW = 4;                                    // stages of operands as they come
    static constexpr int ACC = NX == 96 ? 1 : NX == 16 ? 4 : 2;       // accumulators of a slab's large products
    static constexpr int SPLIT = NX == 64 ? 4 : NX == 16 ? 3 : 2;    // stages of split operands (W: tensor memory, x: shared memory)
    static constexpr int TMEM = NX <= 32 ? 256 : 512;                // columns: the accumulators, three more for a part's small products, 48 per split stage
    static constexpr int S_COL = ACC * NX, A_COL = S_COL + 3 * NX;
    static constexpr int SX_BYTES = NX * 64;                         // a part of x
    static constexpr int BLOCKS = NX <= 32 ? 2 : 1;
    // Warps that split x.  Where registers run out (the adding warps hold up to 96 sums a thread), warpgroups trade them: 640 threads start
    // with 96 each, the adding 256 take GROW and the other 384 keep SHRINK (256 GROW + 384 SHRINK <= 640 x 96).
    // The pool may be just as large as what is asked for, so nobody takes registers back before the adding warps are through with
    // theirs: a barrier of all warps (of the cluster, or of the block alone) stands between every warp's first trade and its second, and behind it
    // the adding warps give back without waiting for anything.
    static constexpr int X_WARP = NX >= 64 ? 16 : 14, X_WARPS = NX >= 64 ? 4 : 2, THREADS = 32 * (X_WARP + X_WARPS);
    static constexpr int START = 96, GROW = NX >= 96 ? 168 : 136, SHRINK = NX >= 96 ? 48 : 64;
    static constexpr bool SHIFT_REGS = NX >= 64;
    static_assert(!SHIFT_REGS || (THREADS == 640 && 256 * GROW + 384 * SHRINK <= 640 * START && 640 * START <= 65536), "registers");
    static constexpr int TILES = RAW * (A_BYTES + X_BYTES) + SPLIT * 3 * SX_BYTES;
    static_assert(A_COL + 48 * SPLIT <= TMEM, "tensor memory");
};

struct SpShared {
    uint64_t raw_full[4], raw_empty[4], split_full[4], split_empty[4], acc_full[4], acc_empty[4], small_full, small_empty;
    uint32_t tmem_base;
    int large_w[SP_TILE_W], large_x[96];         // rows' largest finite values where they exceed SP_LARGE, as the bits of floats
};

struct SpArgs {
    const float* A;
    const float* W;
    float* C;
    int M, N, K, xt, tma, w_batched, x_batched;
    int64_t lda, ldw, ldc, sa, sw, sc;
    int* status;
};

// bfloat16 products: A from tensor memory (a column per two values of k), B from shared memory
__device__ __forceinline__ void sp_mma(uint32_t tmem_d, uint32_t tmem_a, uint64_t desc_b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(tmem_d), "r"(tmem_a), "l"(desc_b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void sp_st8(uint32_t taddr, const uint32_t* v) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};"
                 ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]));
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
// Shared-memory matrix descriptor of a K-major tile with 64-byte swizzle: rows of 64 bytes, 8-row groups 512 bytes apart.
__device__ __forceinline__ uint64_t sp_desc(uint32_t smem_addr) {
    const uint32_t lo = ((smem_addr >> 4) & 0x3FFFu) | (1u << 16);
    const uint32_t hi = 32u | (1u << 14) | (4u << 29);
    return ((uint64_t)hi << 32) | lo;
}
// Two values as three bfloat16 each, x = a + b + c exactly: x rounded, what is left of it rounded, and the rest
__device__ __forceinline__ void sp_split2(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    auto pack = [&](uint32_t& to) { asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(to) : "f"(y), "f"(x)); };       // (x in the lower half)
    auto less = [&](uint32_t by) {
        x -= __uint_as_float(by << 16);
        y -= __uint_as_float(by & 0xffff0000u);
    };
    pack(a);
    less(a);
    pack(b);
    less(b);
    pack(c);
}
#define SP_LARGE 0x1p20f
__device__ __forceinline__ float sp_larger(float m, float x) { return fmaxf(m, fabsf(x)); }       // (results of rows with infinities are computed again anyhow)

// One output as a chain of multiply-adds over k = 0, 1, ...
__device__ __noinline__ float sp_chain(const float* a, const float* w, int K) {
    float acc = 0.f;
    for (int k = 0; k < K; ++k) acc = fmaf(a[k], w[k], acc);
    return acc;
}
// Whether a result is computed again, given the large values of its two rows.  A value's parts end at 2^-136 (at 2^-126 if the unit took small ones for
// zeros), so a sum of K products with values up to L in the other row may be off by K L 2^-125, and from L 2^-80 on that is nothing.
__device__ __forceinline__ bool sp_irregular(float v, int large_w, int large_x) {
    const float a = fabsf(v), large = __int_as_float(max(large_w, large_x));
    return !(a < INFINITY) || (a < fmaxf(0x1p-60f, large * 0x1p-80f) && (a != 0.f || large > 0.f));
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
    constexpr int COLS = NX / 2, OWN = SP_PARTS / CL, RAW = Cfg::RAW, SPLIT = Cfg::SPLIT, ACC = Cfg::ACC;
    constexpr int LD = COLS % 16 == 0 ? 16 : 8;
    extern __shared__ unsigned char sp_dyn[];
    unsigned char* base = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(sp_dyn) + 1023) & ~(uintptr_t)1023);
    unsigned char* raw_w = base;                                        // [stage][128 rows][128 bytes], 128-byte swizzle
    unsigned char* raw_x = raw_w + RAW * Cfg::A_BYTES;                  // [stage][NX rows][128 bytes]
    unsigned char* split_x = raw_x + RAW * Cfg::X_BYTES;                // [stage][a, b, c][NX rows][64 bytes], 64-byte swizzle
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
            mbar_init(&sh->split_empty[s], 1);
        }
        for (int b = 0; b < ACC; ++b) {
            mbar_init(&sh->acc_full[b], 1);
            mbar_init(&sh->acc_empty[b], 8);
        }
        mbar_init(&sh->small_full, 1);
        mbar_init(&sh->small_empty, 8);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (threadIdx.x < SP_TILE_W) sh->large_w[threadIdx.x] = 0;
    if (threadIdx.x < NX) sh->large_x[threadIdx.x] = 0;
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
    // the splitting warps have looked at every value: what they noted may be read by the adding warps of their block
    constexpr int SPLITTERS = 32 * (4 + Cfg::X_WARPS);
    auto noted = [&]() {
        __syncwarp();
        if (CL == 1) asm volatile("bar.arrive 2, %0;" ::"n"(256 + SPLITTERS) : "memory");
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
        int parts = 0;
        // a part's n slabs, one after the other, then its small products
        auto add_part = [&](float (&to)[COLS], int n) {
            for (int i = 0; i < n; ++i, acc.next(ACC)) {
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
            if (n <= 0) return;
            wait(&sh->small_full, parts & 1, 20);
            ++parts;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < COLS; c0 += 8) {
                uint32_t r[3][8];
#pragma unroll
                for (int o = 0; o < 3; ++o) sp_ld8(trow + Cfg::S_COL + o * NX + c0, r[o]);
                asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                if (c0 + 8 >= COLS) {
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&sh->small_empty);
                }
#pragma unroll
                for (int c = 0; c < 8; ++c) to[c0 + c] += __uint_as_float(r[0][c]) + (__uint_as_float(r[1][c]) + __uint_as_float(r[2][c]));
            }
        };
        pdl_wait();
        if constexpr (CL > 1) {
#pragma unroll
            for (int p = 0; p < OWN; ++p) add_part(sum[p], max(0, min(slabs, (rank * OWN + p + 1) * part) - min(slabs, (rank * OWN + p) * part)));
            if (!ok)
#pragma unroll
                for (int c = 0; c < COLS; ++c) sum[0][c] = INFINITY;
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
            __syncwarp();
            asm volatile("bar.sync 2, %0;" ::"n"(256 + SPLITTERS) : "memory");
            const int large = sh->large_w[quarter * 32 + lane], n = n0 + quarter * 32 + lane;
            if (n < a.N) {
                const float* w = a.W + (int64_t)z * a.sw + (int64_t)n * a.ldw;
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    const int m = m0 + half * COLS + c;
                    if (m < a.M) {
                        float v = ok ? sum[0][c] : INFINITY;          // (after a wait that ran out: as for results that are not finite)
                        if (sp_irregular(v, large, sh->large_x[half * COLS + c])) v = sp_chain(a.A + (int64_t)z * a.sa + (int64_t)m * a.lda, w, a.K);
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
            constexpr int AHEAD = NX >= 96 ? 1 : 2;        // groups of 16 values read ahead: as many as the registers hold
            Ring raw, split;
            float largest = 0.f;
            for (int it = 0; it < last - first; ++it, raw.next(RAW), split.next(SPLIT)) {
                wait(&sh->raw_full[raw.at], raw.round, 21);
                if (!ok) break;
                const unsigned char* src = raw_w + raw.at * Cfg::A_BYTES + row * 128;
                float4 v[AHEAD][4];
                auto load = [&](int g) {
#pragma unroll
                    for (int c = 0; c < 4; ++c) v[g % AHEAD][c] = *reinterpret_cast<const float4*>(src + (((4 * g + c) ^ (row & 7)) << 4));
                };
#pragma unroll
                for (int g = 0; g < AHEAD; ++g) load(g);
                if (it >= SPLIT) {
                    wait(&sh->split_empty[split.at], split.round ^ 1, 22);
                    if (!ok) break;
                    tc_fence_after();
                }
#pragma unroll
                for (int g = 0; g < 2; ++g) {
                    uint32_t part[3][8];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const float4 q = v[g % AHEAD][c];
                        largest = sp_larger(sp_larger(sp_larger(sp_larger(largest, q.x), q.y), q.z), q.w);
                        sp_split2(q.x, q.y, part[0][2 * c], part[1][2 * c], part[2][2 * c]);
                        sp_split2(q.z, q.w, part[0][2 * c + 1], part[1][2 * c + 1], part[2][2 * c + 1]);
                    }
                    if (g + AHEAD < 2) load(g + AHEAD);
#pragma unroll
                    for (int p = 0; p < 3; ++p) sp_st8(tlane + split.at * 48 + 16 * p + 8 * g, part[p]);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->raw_empty[raw.at]);
                asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(&sh->split_full[split.at]);
            }
            if (largest > SP_LARGE) sh->large_w[row] = __float_as_int(largest);
            noted();
        } else if (warp >= Cfg::X_WARP) {
            constexpr int XT = 32 * Cfg::X_WARPS;
            const int t = threadIdx.x - Cfg::X_WARP * 32;
            constexpr int PIECES = NX * 4 / XT;      // of a thread: 8 values of a row each
            static_assert(PIECES * XT == NX * 4, "pieces");
            Ring raw, split;
            for (int it = 0; it < last - first; ++it, raw.next(RAW), split.next(SPLIT)) {
                wait(&sh->raw_full[raw.at], raw.round, 23);
                if (it >= SPLIT) wait(&sh->split_empty[split.at], split.round ^ 1, 24);
                if (!ok) break;
                const unsigned char* src = raw_x + raw.at * Cfg::X_BYTES;
                unsigned char* dst = split_x + split.at * 3 * Cfg::SX_BYTES;
#pragma unroll
                for (int i = 0; i < PIECES; ++i) {
                    const int r = (t + XT * i) >> 2, u = t & 3;
                    const float4 v = *reinterpret_cast<const float4*>(src + r * 128 + (((2 * u) ^ (r & 7)) << 4));
                    const float4 w = *reinterpret_cast<const float4*>(src + r * 128 + (((2 * u + 1) ^ (r & 7)) << 4));
                    const float largest = sp_larger(sp_larger(sp_larger(fabsf(v.x), v.y), sp_larger(fabsf(v.z), v.w)), sp_larger(sp_larger(fabsf(w.x), w.y), sp_larger(fabsf(w.z), w.w)));
                    if (largest > SP_LARGE) atomicMax(&sh->large_x[r], __float_as_int(largest));
                    uint32_t part[3][4];
                    sp_split2(v.x, v.y, part[0][0], part[1][0], part[2][0]);
                    sp_split2(v.z, v.w, part[0][1], part[1][1], part[2][1]);
                    sp_split2(w.x, w.y, part[0][2], part[1][2], part[2][2]);
                    sp_split2(w.z, w.w, part[0][3], part[1][3], part[2][3]);
#pragma unroll
                    for (int p = 0; p < 3; ++p)
                        *reinterpret_cast<uint4*>(dst + p * Cfg::SX_BYTES + r * 64 + ((u ^ ((r >> 1) & 3)) << 4)) = make_uint4(part[p][0], part[p][1], part[p][2], part[p][3]);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive(&sh->raw_empty[raw.at]);
                    mbar_arrive(&sh->split_full[split.at]);
                }
            }
            noted();
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
            // instruction descriptor: f32 accumulate, bfloat16 operands, both K-major, M = 128, N = n
            constexpr auto idesc = [](int n) { return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | ((128u >> 4) << 24); };
            // One thread issues; the next slab's operands are waited for ahead of a slab's last products, so that the unit's queue does not run dry.
            // The parts of x that meet a part of W stand one behind the other in shared memory, and their results in tensor memory: by size
            // a's b and b's a, then a's c, b's b and c's a, then b's c and c's b.
            uint32_t leader = 0;
            asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(leader));
            if (leader) {
                Ring acc, split, ahead;
                int parts = 0;
                auto operands = [&](int it) {
                    if (it >= last - first) return;
                    ok = ok && passed(&sh->split_full[ahead.at], ahead.round, 27);
                    ahead.next(SPLIT);
                };
                operands(0);
                for (int it = 0; it < last - first && ok; ++it, acc.next(ACC), split.next(SPLIT)) {
                    const bool opens = it % part == 0, closes = it % part == part - 1 || it == last - first - 1;
                    const uint32_t small = tmem + Cfg::S_COL, wa = tmem + Cfg::A_COL + split.at * 48, wb = wa + 16, wc = wb + 16;
                    const uint32_t xa = tc_smem(split_x + split.at * 3 * Cfg::SX_BYTES), xb = xa + Cfg::SX_BYTES, xc = xb + Cfg::SX_BYTES;
                    auto large = [&]() {
                        if (it >= ACC) ok = ok && passed(&sh->acc_empty[acc.at], acc.round ^ 1, 26);
                        if (!ok) return;
                        tc_fence_after();
#pragma unroll
                        for (int k = 0; k < 2; ++k) sp_mma(tmem + acc.at * NX, wa + 8 * k, sp_desc(xa + 32 * k), idesc(NX), k > 0 ? 1u : 0u);
                        tc_commit(&sh->acc_full[acc.at]);
                    };
                    tc_fence_after();
                    if (opens) {            // (the adding warps come to the last part's small products behind its large ones)
                        large();
                        if (it > 0) ok = ok && passed(&sh->small_empty, (parts - 1) & 1, 26);
                        if (!ok) break;
                        tc_fence_after();
                        ++parts;
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) {
                        const uint32_t add = !opens || k > 0 ? 1u : 0u;
                        if constexpr (3 * NX <= 256) sp_mma(small, wb + 8 * k, sp_desc(xa + 32 * k), idesc(3 * NX), add);
                        else {
                            sp_mma(small, wb + 8 * k, sp_desc(xa + 32 * k), idesc(2 * NX), add);
                            sp_mma(small + 2 * NX, wb + 8 * k, sp_desc(xc + 32 * k), idesc(NX), add);
                        }
                    }
#pragma unroll
                    for (int k = 0; k < 2; ++k) sp_mma(small, wa + 8 * k, sp_desc(xb + 32 * k), idesc(2 * NX), 1u);
                    if (opens) operands(it + 1);
#pragma unroll
                    for (int k = 0; k < 2; ++k) sp_mma(small + NX, wc + 8 * k, sp_desc(xa + 32 * k), idesc(2 * NX), 1u);
                    if (!opens) {
                        operands(it + 1);
                        large();
                    }
                    if (closes) tc_commit(&sh->small_full);
                    tc_commit(&sh->split_empty[split.at]);
                }
            }
            __syncwarp();
        }
        if (CL > 1) {
            __syncwarp();
            asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
            asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
            // a block knows the large values of its own parts of K: every block of the cluster gets them (there are hardly ever any)
            for (int i = threadIdx.x - 256; i < SP_TILE_W + NX; i += Cfg::THREADS - 256) {
                int* at = i < SP_TILE_W ? &sh->large_w[i] : &sh->large_x[i - SP_TILE_W];
                const int large = *at;
                for (int r = 0; large != 0 && r < CL; ++r)
                    asm volatile("red.relaxed.cluster.shared::cluster.max.s32 [%0], %1;" ::"r"(cluster_addr(tc_smem(at), r)), "r"(large) : "memory");
            }
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
                if (sp_irregular(v, sh->large_w[rank * SHARE + l], sh->large_x[c])) v = sp_chain(a.A + (int64_t)z * a.sa + (int64_t)m * a.lda, a.W + (int64_t)z * a.sw + (int64_t)n * a.ldw, a.K);
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
// and the slabs a block walks (measured at K 512 to 6,144, 1 to 2,048 rows, nine sizes of W from memory; a slab is 128 x NX x 32):
//   rows of x       16     32     64     96
//   per slab       0.52   0.66   0.64   0.87   (16 and 32: two blocks fit a multiprocessor, and take 0.3 to 0.5 each when they share it; one block
//                                              that walks all of K, many of which stream W from memory: 0.60 and 0.70)
//   start, end      5.2    5.0    9.2   12.7    one block walks K;  4.3 to 6.4 in a cluster
// so 96 rows of x per tile are the cheapest per output, fewer where they leave padding, and a cluster pays where tiles leave
// multiprocessors idle.  (Clusters of 8, and of 2 or 4 blocks that may share a multiprocessor, do not reach all of them: 16 clusters of 8 one to
// a multiprocessor take two rounds, 14 take one.)  Of 117 products its choice is the fastest or within 10 % of it at 111, within 30 % at the rest.
struct SpForm {
    int nx, cl;
    float slab, shared, ends;
};
static const SpForm SP_FORMS[] = {
    {16, 1, 0.60f, 0.34f, 5.2f}, {16, 2, 0.52f, 0.37f, 5.5f}, {16, 4, 0.52f, 0.36f, 5.5f}, {16, 8, 0.52f, 0.27f, 4.3f}, {32, 1, 0.70f, 0.50f, 5.0f},
    {32, 4, 0.66f, 0.57f, 6.0f}, {32, 8, 0.66f, 0.45f, 5.1f}, {64, 1, 0.61f, 0.f, 9.2f}, {64, 4, 0.64f, 0.f, 6.4f}, {64, 8, 0.64f, 0.f, 5.5f},
    {96, 1, 0.83f, 0.f, 12.7f},
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
    }
    X0NE_REQUIRE(false, "gemm_f32: no form %d for M %d N %d", form, M, N);
}
