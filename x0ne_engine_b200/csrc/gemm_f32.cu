// C[M,N] = A[M,K] * W[N,K]^T in true float32: FMA on the CUDA cores, no tensor-core mode.
//
// This is the matrix product of the 32-bit path where K is below 512 (longer ones: gemm_f32_tcgen05.cu).  Each output is ONE chain of fused
// multiply-adds over k = 0, 1, ..., K-1 in that order, whatever M is and wherever the output
// lies in its tile, so a row's result is bit-identical whether the row is computed alone, in a
// batch, in a prompt or in a decode step.  (The library engine calls cublasGemmEx for its
// products, x0ne-core/runtime/src/gpu.rs:1098-1149; a library picks its algorithm by shape, so
// the same row can round differently at different M, which this kernel exists to rule out.)
//
// Tile 128 x 64 x 16, 256 threads, 8 x 4 outputs per thread, operands staged through shared
// memory with the k index outermost.
#include "common.cuh"

#define BM 128
#define BN 64
#define BK 16
#define TM 8
#define TN 4

__global__ void __launch_bounds__(256) gemm_f32_nt_kernel(const float* A, const float* W,
                                                           float* __restrict__ C, int M, int N, int K, int lda,
                                                           int ldw, int ldc, int64_t sa, int64_t sw, int64_t sc) {
    __shared__ float As[BK][BM + 4];
    __shared__ float Ws[BK][BN + 4];
    pdl_prologue();
    A += blockIdx.z * sa;       // one product per z: a batch of independent products of one shape
    W += blockIdx.z * sw;
    C += blockIdx.z * sc;
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;  // tx: 16 column groups of 4, ty: 16 row groups of 8
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;

    for (int k0 = 0; k0 < K; k0 += BK) {
        // A tile: 128 rows x 16 k = 2048 values, 8 per thread
#pragma unroll
        for (int it = 0; it < 8; ++it) {
            const int idx = tid + it * 256;
            const int r = idx / BK, kk = idx % BK;
            const int gm = m0 + r, gk = k0 + kk;
            As[kk][r] = (gm < M && gk < K) ? A[(int64_t)gm * lda + gk] : 0.f;
        }
        // W tile: 64 rows x 16 k = 1024 values, 4 per thread
#pragma unroll
        for (int it = 0; it < 4; ++it) {
            const int idx = tid + it * 256;
            const int r = idx / BK, kk = idx % BK;
            const int gn = n0 + r, gk = k0 + kk;
            Ws[kk][r] = (gn < N && gk < K) ? W[(int64_t)gn * ldw + gk] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], b[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) b[j] = Ws[kk][tx * TN + j];
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int gm = m0 + ty * TM + i;
        if (gm >= M) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int gn = n0 + tx * TN + j;
            if (gn < N) C[(int64_t)gm * ldc + gn] = acc[i][j];
        }
    }
}

// The same chains for operands that can be read 16 bytes at a time (K, strides and bases multiples of four values).
//
// Many rows: a tile of BM x BN outputs, TM x TN per thread (its rows and columns in pieces of four, so that a warp's 16-byte reads of shared
// memory meet no bank twice), 16 values of k at a time in two buffers, the next ones on their way to registers meanwhile; with AHEAD
// the next k's values are read while the current one's products are made.  100 / 200 / 400 rows against W 1024 x 256 take 9.7 / 11.0 / 19.2 us,
// 4096 x 256 18.8 / 32.1 / 35.3: waits for shared memory and between dependent multiply-adds, not the units' rate.
template <int BM_, int BN_, int TM_, int TN_, bool AHEAD, int BLOCKS>
__global__ void __launch_bounds__(BM_ / TM_ * (BN_ / TN_), BLOCKS) gemm_f32_tile_kernel(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda,
                                                                               int64_t ldw, int64_t ldc, int64_t sa, int64_t sw, int64_t sc) {
    constexpr int KT = 16, THREADS = BM_ / TM_ * (BN_ / TN_), TX = BN_ / TN_;
    constexpr int AQ = BM_ * KT / 4 / THREADS, WQ = BN_ * KT / 4 / THREADS;      // 16-byte pieces of each operand per thread and step
    static_assert(AQ * THREADS * 4 == BM_ * KT && WQ * THREADS * 4 == BN_ * KT && TM_ % 4 == 0 && TN_ % 4 == 0, "tile");
    __shared__ __align__(16) float As[2][KT][BM_ + 4], Ws[2][KT][BN_ + 4];
    pdl_prologue();
    A += blockIdx.z * sa;
    W += blockIdx.z * sw;
    C += blockIdx.z * sc;
    const int tid = threadIdx.x, tx = tid % TX, ty = tid / TX;
    const int m0 = blockIdx.y * BM_, n0 = blockIdx.x * BN_;
    float acc[TM_][TN_];
#pragma unroll
    for (int i = 0; i < TM_; ++i)
#pragma unroll
        for (int j = 0; j < TN_; ++j) acc[i][j] = 0.f;
    float4 fa[AQ], fw[WQ];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < AQ; ++i) {
            const int e = tid + i * THREADS, r = m0 + e / (KT / 4), k = k0 + e % (KT / 4) * 4;
            fa[i] = r < M && k < K ? *reinterpret_cast<const float4*>(A + r * lda + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < WQ; ++i) {
            const int e = tid + i * THREADS, r = n0 + e / (KT / 4), k = k0 + e % (KT / 4) * 4;
            fw[i] = r < N && k < K ? *reinterpret_cast<const float4*>(W + r * ldw + k) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](int b) {
#pragma unroll
        for (int i = 0; i < AQ; ++i) {
            const int e = tid + i * THREADS, r = e / (KT / 4), k = e % (KT / 4) * 4;
            As[b][k][r] = fa[i].x; As[b][k + 1][r] = fa[i].y; As[b][k + 2][r] = fa[i].z; As[b][k + 3][r] = fa[i].w;
        }
#pragma unroll
        for (int i = 0; i < WQ; ++i) {
            const int e = tid + i * THREADS, r = e / (KT / 4), k = e % (KT / 4) * 4;
            Ws[b][k][r] = fw[i].x; Ws[b][k + 1][r] = fw[i].y; Ws[b][k + 2][r] = fw[i].z; Ws[b][k + 3][r] = fw[i].w;
        }
    };
    __align__(16) float a[2][TM_], w[2][TN_];
    auto read = [&](int b, int kk, int q) {
#pragma unroll
        for (int i = 0; i < TM_; i += 4) *reinterpret_cast<float4*>(&a[q][i]) = *reinterpret_cast<const float4*>(&As[b][kk][i / 4 * (BM_ * 4 / TM_) + ty * 4]);
#pragma unroll
        for (int j = 0; j < TN_; j += 4) *reinterpret_cast<float4*>(&w[q][j]) = *reinterpret_cast<const float4*>(&Ws[b][kk][j / 4 * (BN_ * 4 / TN_) + tx * 4]);
    };
    fetch(0);
    put(0);
    __syncthreads();
    int b = 0;
    if (AHEAD) read(0, 0, 0);
    for (int k0 = 0; k0 < K; k0 += KT, b ^= 1) {
        const bool more = k0 + KT < K;
        if (more) fetch(k0 + KT);
#pragma unroll
        for (int kk = 0; kk < KT; ++kk) {
            const int q = AHEAD ? kk & 1 : 0;
            if (!AHEAD) read(b, kk, 0);
            else if (kk + 1 < KT) read(b, kk + 1, q ^ 1);
            else {
                if (more) put(b ^ 1);
                __syncthreads();
                if (more) read(b ^ 1, 0, q ^ 1);
            }
#pragma unroll
            for (int i = 0; i < TM_; ++i)
#pragma unroll
                for (int j = 0; j < TN_; ++j) acc[i][j] = fmaf(a[q][i], w[q][j], acc[i][j]);
        }
        if (!AHEAD) {
            if (more) put(b ^ 1);
            __syncthreads();
        }
    }
    const bool vec = ldc % 4 == 0 && (((uintptr_t)C) & 15) == 0;
#pragma unroll
    for (int i = 0; i < TM_; ++i) {
        const int m = m0 + i / 4 * (BM_ * 4 / TM_) + ty * 4 + i % 4;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < TN_; j += 4) {
            const int n = n0 + j / 4 * (BN_ * 4 / TN_) + tx * 4;
            float* c = C + m * ldc + n;
            if (vec && n + 3 < N) *reinterpret_cast<float4*>(c) = make_float4(acc[i][j], acc[i][j + 1], acc[i][j + 2], acc[i][j + 3]);
            else
#pragma unroll
                for (int q = 0; q < 4; ++q)
                    if (n + q < N) c[q] = acc[i][j + q];
        }
    }
}

// Few rows (at most 4 RM).  A block takes 32 outputs of every row, a thread one of them for RM rows; W's rows and x stream through a ring of
// copies, FEW_K values of k a stage, and are read along k.  8 rows against W 1024 x 256 / 4096 x 256 take 3.5 / 4.3 us, 64 rows 9.6 / 12.7; bound by
// a block's walk along k, not by the bytes of W.
#define FEW_K 64
#define FEW_STAGES 4
__device__ __forceinline__ void few_copy16(float* dst, const float* src, bool ok) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(n) : "memory");
}
template <int RM>
__global__ void __launch_bounds__(128) gemm_f32_few_kernel(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc,
                                                           int64_t sa, int64_t sw, int64_t sc) {
    constexpr int PITCH = FEW_K + 4;         // (a warp's 16-byte reads of 32 rows meet every bank once per eight lanes)
    extern __shared__ __align__(16) float few_smem[];
    float* Ws = few_smem;                                          // [stage][32][PITCH]
    float* Xs = few_smem + FEW_STAGES * 32 * PITCH;                // [stage][4 RM][PITCH]
    pdl_launch_dependents();
    const int tid = threadIdx.x, n = tid & 31, mg = tid >> 5, n0 = blockIdx.x * 32;
    A += blockIdx.z * sa;
    W += blockIdx.z * sw;
    C += blockIdx.z * sc;
    const int steps = (K + FEW_K - 1) / FEW_K;
    pdl_wait();         // (W may be a product's result too)
    auto issue = [&](int step) {
        if (step < steps) {
            const int st = step % FEW_STAGES, k0 = step * FEW_K;
#pragma unroll
            for (int i = 0; i < 32 * FEW_K / 4 / 128; ++i) {
                const int e = tid + i * 128, r = e / (FEW_K / 4), k = e % (FEW_K / 4) * 4;
                const bool ok = n0 + r < N && k0 + k < K;
                few_copy16(Ws + (st * 32 + r) * PITCH + k, ok ? W + (n0 + r) * ldw + k0 + k : W, ok);
            }
#pragma unroll
            for (int i = 0; i < (4 * RM * FEW_K / 4 + 127) / 128; ++i) {
                const int e = tid + i * 128, r = e / (FEW_K / 4), k = e % (FEW_K / 4) * 4;
                const bool ok = r < M && k0 + k < K;
                if (r < 4 * RM) few_copy16(Xs + (st * 4 * RM + r) * PITCH + k, ok ? A + r * lda + k0 + k : A, ok);
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int i = 0; i < FEW_STAGES - 1; ++i) issue(i);
    float acc[RM];
#pragma unroll
    for (int i = 0; i < RM; ++i) acc[i] = 0.f;
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FEW_STAGES - 2) : "memory");
        __syncthreads();            // this step's copies have landed for every thread, and the stage before is no longer read
        issue(step + FEW_STAGES - 1);
        const float* w = Ws + (step % FEW_STAGES * 32 + n) * PITCH;
        const float* x = Xs + (step % FEW_STAGES * 4 * RM + mg * RM) * PITCH;
#pragma unroll
        for (int k = 0; k < FEW_K; k += 4) {
            const float4 w4 = *reinterpret_cast<const float4*>(w + k);
#pragma unroll
            for (int i = 0; i < RM; ++i) {
                const float4 x4 = *reinterpret_cast<const float4*>(x + i * PITCH + k);
                acc[i] = fmaf(x4.x, w4.x, acc[i]);
                acc[i] = fmaf(x4.y, w4.y, acc[i]);
                acc[i] = fmaf(x4.z, w4.z, acc[i]);
                acc[i] = fmaf(x4.w, w4.w, acc[i]);
            }
        }
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    if (n0 + n < N)
#pragma unroll
        for (int i = 0; i < RM; ++i)
            if (mg * RM + i < M) C[(mg * RM + i) * ldc + n0 + n] = acc[i];
}

template <int BM_, int BN_, int TM_, int TN_, bool AHEAD, int BLOCKS>
static void gemm_f32_tiles(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch, int64_t sa, int64_t sw, int64_t sc,
                           cudaStream_t stream) {
    x0ne_launch(gemm_f32_tile_kernel<BM_, BN_, TM_, TN_, AHEAD, BLOCKS>, dim3((N + BN_ - 1) / BN_, (M + BM_ - 1) / BM_, batch), dim3(BM_ / TM_ * (BN_ / TN_)), 0, stream, A, W, C, M, N, K,
                lda, ldw, ldc, sa, sw, sc);
}
template <int RM>
static int gemm_f32_few(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc, int batch, int64_t sa, int64_t sw, int64_t sc,
                        cudaStream_t stream) {
    const size_t smem = (size_t)FEW_STAGES * (32 + 4 * RM) * (FEW_K + 4) * sizeof(float);
    static OncePerDevice configured;
    if (configured.need()) {
        cudaError_t e = cudaFuncSetAttribute(gemm_f32_few_kernel<RM>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        X0NE_REQUIRE(e == cudaSuccess, "gemm_f32: %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
        configured.done();
    }
    x0ne_launch(gemm_f32_few_kernel<RM>, dim3((N + 31) / 32, 1, batch), dim3(128), smem, stream, A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc);
    return 0;
}

extern "C" int x0ne_gemm_f32_split(const float* A, const float* W, float* C, int M, int N, int K, int64_t lda, int64_t ldw, int64_t ldc, int batch, int64_t sa, int64_t sw, int64_t sc,
                                   int form, int* status, cudaStream_t stream);       // gemm_f32_tcgen05.cu

// K from which the tensor cores take a product.  The rule may look at W alone, so that a row's bits do not depend on what is computed with
// it.  8 / 64 rows on multiply-add units against tensor cores: K 512 7.0 / 24.6 us and 7.5 / 10.2 (N 4096), 6.4 / 17.2 and 6.3 / 6.8 (N 1024); K 1,024 10.8 /
// 31.5 and 6.5 / 8.1 (N 1024); K 2,048 24.4 / 89 and 13.3 / 18.6 (N 4096); K 256 6.9 / 13.6 and 9.2 / 8.9 (N 4096), 7.4 / 10.0 and 8.7 / 8.8 (N 1024).
// Their error against 64 bits is the smaller one for dense rows (2-norm over 2-norm, multiply-adds and tensor cores: K 256 2.9e-7 and 7.3e-8, 512 4.1e-7
// and 7.8e-8, 2,048 8.2e-7 and 9.2e-8, 6,144 1.4e-6 and 1.2e-7; all values positive 3.3e-7 and 5.9e-8 at 512, 1.2e-6 and 6.8e-8 at 6,144), and about the same where
// a row has a handful of terms (one value in a hundred not zero: 4.7e-8 and 4.9e-8 at 512, 8.4e-8 and 6.0e-8 at 2,048).
#define F32_SPLIT_K 512

// `batch` products of one shape: product b reads A + b sa and W + b sw and writes C + b sc.  `status`: one int in device memory, zero before the
// first call (a wait of the tensor-core kernel that ran out leaves a bit there).
X0NE_API int x0ne_gemm_f32_nt_batched(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                                      int batch, int64_t sa, int64_t sw, int64_t sc, int* status, cudaStream_t stream) {
    X0NE_REQUIRE(M >= 0 && N > 0 && K > 0 && lda >= K && ldw >= K && ldc >= N, "gemm_f32: M %d N %d K %d lda %d ldw %d ldc %d",
                 M, N, K, lda, ldw, ldc);
    X0NE_REQUIRE(batch >= 1 && batch <= 65535, "gemm_f32: batch %d", batch);
    if (M == 0) return 0;
    if (K >= F32_SPLIT_K) return x0ne_gemm_f32_split(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, 0, status, stream);
    if (K % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && sa % 4 == 0 && sw % 4 == 0 && ((((uintptr_t)A) | ((uintptr_t)W)) & 15) == 0 && M <= 64 * 65535) {
        if (M <= 8) {
            if (int e = gemm_f32_few<2>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream)) return e;
        } else if (M <= 16) {
            if (int e = gemm_f32_few<4>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream)) return e;
        } else if (M <= 32) {
            if (int e = gemm_f32_few<8>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream)) return e;
        } else if (M <= 64 && N <= 8192) {
            if (int e = gemm_f32_few<16>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream)) return e;
        } else {
            // the largest tile that still gives every multiprocessor several (64 x 128), one (64 x 64), else small ones (measured at K 2,048, where all
            // three still ran: 64 x 128 / 64 x 64 / 32 x 64 at 3,072 tiles of 64 x 128 2288 / 2600 / 3225 us, at 512 572 / 440 / 547, at 32 161 / 99 / 70)
            const int64_t m64 = (M + 63) / 64, m32 = (M + 31) / 32, sms = x0ne_sm_count();
            if (batch * m64 * ((N + 127) / 128) >= 6 * sms) gemm_f32_tiles<64, 128, 8, 8, false, 1>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
            else if (batch * m64 * ((N + 63) / 64) >= sms || m32 > 65535) gemm_f32_tiles<64, 64, 4, 8, true, 4>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
            else gemm_f32_tiles<32, 64, 4, 4, true, 1>(A, W, C, M, N, K, lda, ldw, ldc, batch, sa, sw, sc, stream);
        }
        X0NE_LAUNCH_CHECK();
    }
    dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    X0NE_REQUIRE(grid.y <= 65535, "gemm_f32: M %d needs more than 65535 row tiles", M);
    x0ne_launch(gemm_f32_nt_kernel, dim3(grid), dim3(256), 0, stream, A, W, C, M, N, K, lda, ldw, ldc, sa, sw, sc);
    X0NE_LAUNCH_CHECK();
}

X0NE_API int x0ne_gemm_f32_nt(const float* A, const float* W, float* C, int M, int N, int K, int lda, int ldw, int ldc,
                              int* status, cudaStream_t stream) {
    return x0ne_gemm_f32_nt_batched(A, W, C, M, N, K, lda, ldw, ldc, 1, 0, 0, 0, status, stream);
}
