// The matrix-state recurrence of wkv.cu for long runs of tokens in bfloat16: by chunks of 64 tokens, all chunks at once.
//
//   out_t = r_t (S + u k_t v_t),  S <- w_t S + k_t v_t   per head, with S [64 key channels][64 value channels], w_t = exp(-exp(z_t + w0))
// The token-by-token kernel is one chain through a sequence, and its 128 blocks at 32 heads use half of their issue slots: 70 ns a token.
// With P(a, b) the product of the decays of the tokens a .. b (1 where there are none), a chunk that starts from S gives
//   out_t = (r_t P(first, t - 1)) S + sum_{s < t} A[t][s] v_s + A[t][t] v_t,   A[t][s] = sum_i r_t k_s P(s + 1, t - 1),   A[t][t] = sum_i r_t u k_t
//   S'    = P(first, last) S + sum_s (k_s P(s + 1, last)) v_s
// so the chunks' own terms need no state, and the states follow one another by one multiply-add per value and chunk:
//   wkv_chunk_sums     per (chunk, head): B = sum_s (k_s P(s + 1, last)) v_s and P(first, last)
//   wkv_chunk_states   per value of a head's state, chunk after chunk: B is replaced by the state that the chunk starts from
//   wkv_chunk_out      per (chunk, head): the outputs
// Decays are products of numbers in [0, 1], taken inside blocks of 8 tokens and over whole blocks, never quotients or differences of
// logarithms: nothing overflows, a factor that underflows belongs to a term that does, and a product of n decays is off by n roundings, as in
// the token-by-token kernel.  Inside a block of 8 tokens A is made by multiply-adds over running products; everything else is a
// product of matrices on mma.sync m16n8k8 with every float32 operand as two TF32 numbers (hi hi + hi lo + lo hi; v is exact as one), float32 sums.
// States, decays and sums are float32.  The order of sums differs from the token-by-token kernels', which stay for 32-bit runs, steps and short runs.
// Infinities and NaN have no two halves (a NaN can even lose itself in the rounding): where a chunk of a head meets one, its products are
// made by multiply-adds of the whole values instead, so that it reaches what it reaches in the token-by-token kernel.
// The scan of one sequence of 2,048 tokens, 32 heads: 148 -> 84 us (sums 20, states 12, outputs 56 each alone), 16 heads 142 -> 54, 64 heads 249 -> 162; 16
// sequences of 128, 32 heads 121 -> 80.  The outputs' kernel, which is most of it, uses 56 % of its issue slots and 57 % of shared memory's
// wavefronts (two blocks of 16 warps a multiprocessor; eight warps with blocks of 16 tokens took 69 us).  Error against float64 (2-norm over 2-norm), walk / chunks: 515 tokens
// with slow decays 8.7e-7 / 8.3e-7, 430 in two sequences with fast ones 1.4e-7 / 1.4e-7, one chunk alone 1.7e-7 / 1.9e-7.
#include "common.cuh"

#define WC_L 64                 // tokens of a chunk
#define WC_B 8                  // tokens of a block
#define WC_BLOCKS (WC_L / WC_B)
#define WC_N 64                 // channels of a head
#define WC_THREADS 512
#define WC_STATE_THREADS 256
#define WC_PITCH_ROW 68         // floats between rows that fragments read along (8 rows x 4 places meet 32 banks)
#define WC_PITCH_COL 72         // and across (4 rows x 8 places)
#define WC_UNIT (WC_N * WC_N + WC_N)         // scratch floats of a chunk and head: B or the state, then the product of its decays

struct WkvChunkArgs {
    const bf16* r;
    const bf16* k;
    const bf16* v;
    const float* z;
    const float* w0;
    const float* u;
    const bf16* h;
    float* o;
    float* state;
    float* scratch;             // [unit][head][WC_UNIT]
    int64_t state_stride;
    const int32_t* seq_first_row;
    const int32_t* seq_slot;
    int32_t heads, width;
};

__device__ __forceinline__ void wc_mma(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// x as two TF32 numbers: rounded (halves away from zero), and what is left
__device__ __forceinline__ void wc_split(float x, uint32_t& hi, uint32_t& lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = (__float_as_uint(x - __uint_as_float(hi)) + 0x1000u) & 0xffffe000u;
}
__device__ __forceinline__ float wc_decay(float z, float w0) { return expf(-expf(z + w0)); }
// where chunk c of a sequence that starts at row0 keeps its scratch (a sequence of n rows has ceil(n / 64) chunks, so no two meet)
__device__ __forceinline__ float* wc_unit(const WkvChunkArgs& a, int seq, int row0, int c, int head) {
    return a.scratch + ((int64_t)(row0 / WC_L + seq + c) * a.heads + head) * WC_UNIT;
}

// Sums of products stay in the tensor core for 16 terms and are added up with rounding from there on (it cuts its sums off).
template <int NT>
__device__ __forceinline__ void wc_add(float (&sum)[NT][4], float (&acc)[NT][4], float (&low)[NT][4]) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            sum[n][e] += acc[n][e] + low[n][e];
            acc[n][e] = low[n][e] = 0.f;
        }
}

// B and the product of decays.  A thread takes one channel of one block of tokens, then a warp 16 key channels x 16 value channels.
__global__ void __launch_bounds__(WC_THREADS, 3) wkv_chunk_sums_kernel(WkvChunkArgs a) {
    __shared__ __align__(16) float kd[WC_L][WC_PITCH_COL], vs[WC_L][WC_PITCH_COL];
    __shared__ float block_decay[WC_BLOCKS][WC_N];
    pdl_launch_dependents();
    const int tid = threadIdx.x, c = blockIdx.x, seq = blockIdx.y, head = blockIdx.z, i = tid % WC_N, b = tid / WC_N;
    const int row0 = a.seq_first_row[seq], t0 = row0 + c * WC_L, nt = min(WC_L, a.seq_first_row[seq + 1] - t0);
    if (a.seq_slot[seq] < 0 || nt <= 0) return;
    const float w0 = a.w0[head * WC_N + i];
    pdl_wait();
    const int64_t ld = (int64_t)a.heads * WC_N, at0 = (int64_t)t0 * ld + (int64_t)head * WC_N + i;
    float w[WC_B], k[WC_B], v[WC_B];
#pragma unroll
    for (int x = 0; x < WC_B; ++x) {
        const int t = b * WC_B + x;
        const int64_t at = at0 + (int64_t)(t < nt ? t : 0) * ld;
        w[x] = a.z[at];
        k[x] = to_f32(a.k[at]);
        v[x] = to_f32(a.v[at]);
    }
    float all = 1.f, odd = 0.f;          // odd: NaN once a value is not finite
#pragma unroll
    for (int x = WC_B - 1; x >= 0; --x) {
        const int t = b * WC_B + x;
        vs[t][i] = t < nt ? v[x] : 0.f;
        odd = fmaf(vs[t][i], 0.f, odd);
        k[x] = t < nt ? k[x] * all : 0.f;                  // (with the decays of the block's later tokens)
        all *= t < nt ? wc_decay(w[x], w0) : 1.f;
    }
    block_decay[b][i] = all;
    __syncthreads();
    float after = 1.f;
#pragma unroll
    for (int x = WC_BLOCKS - 1; x > 0; --x)
        if (x > b) after *= block_decay[x][i];
#pragma unroll
    for (int x = 0; x < WC_B; ++x) {
        kd[b * WC_B + x][i] = k[x] * after;
        odd = fmaf(k[x] * after, 0.f, odd);
    }
    float* unit = wc_unit(a, seq, row0, c, head);
    if (b == 0) unit[WC_N * WC_N + i] = after * all;
    const bool plain = __syncthreads_and(odd == 0.f);
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3, i0 = 16 * (warp & 3), j0 = 16 * (warp >> 2);
    float sum[2][4] = {}, acc[2][4] = {}, low[2][4] = {};
    if (!plain) {
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e)
#pragma unroll 1
                for (int s = 0; s < nt; ++s) sum[n][e] = fmaf(kd[s][i0 + g + 8 * (e >> 1)], vs[s][j0 + 8 * n + 2 * t + (e & 1)], sum[n][e]);
    } else
#pragma unroll
    for (int s = 0; s < WC_L; s += 8) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) wc_split(kd[s + t + 4 * (e >> 1)][i0 + g + 8 * (e & 1)], hi[e], lo[e]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const uint32_t bv[2] = {__float_as_uint(vs[s + t][j0 + 8 * n + g]), __float_as_uint(vs[s + t + 4][j0 + 8 * n + g])};
            wc_mma(acc[n], hi, bv);
            wc_mma(low[n], lo, bv);
        }
        if (s % 16 == 8) wc_add(sum, acc, low);
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e)
            *reinterpret_cast<float2*>(unit + (i0 + g + 8 * e) * WC_N + j0 + 8 * n + 2 * t) = make_float2(sum[n][2 * e], sum[n][2 * e + 1]);
}

// The states that the chunks start from, in the place of their sums; the sequence's state goes on to its last token.  A thread takes four values.
#define WC_AHEAD 8              // chunks read ahead
__global__ void __launch_bounds__(WC_STATE_THREADS) wkv_chunk_states_kernel(WkvChunkArgs a) {
    pdl_prologue();
    const int seq = blockIdx.x, head = blockIdx.y, e = (blockIdx.z * WC_STATE_THREADS + threadIdx.x) * 4, i = e / WC_N;
    const int slot = a.seq_slot[seq], row0 = a.seq_first_row[seq], rows = a.seq_first_row[seq + 1] - row0, chunks = (rows + WC_L - 1) / WC_L;
    if (slot < 0 || rows <= 0) return;
    float* st = a.state + (int64_t)slot * a.state_stride + (int64_t)head * WC_N * WC_N + e;
    float4 s = *reinterpret_cast<const float4*>(st);
    float4 sum[WC_AHEAD];
    float w[WC_AHEAD];
    const int64_t step = (int64_t)a.heads * WC_UNIT;
    float* unit = wc_unit(a, seq, row0, 0, head);
    auto ask = [&](int c, int x) {
        if (c < chunks) {
            sum[x] = *reinterpret_cast<const float4*>(unit + c * step + e);
            w[x] = unit[c * step + WC_N * WC_N + i];
        }
    };
#pragma unroll
    for (int x = 0; x < WC_AHEAD; ++x) ask(x, x);
    for (int c0 = 0; c0 < chunks; c0 += WC_AHEAD) {
#pragma unroll
        for (int x = 0; x < WC_AHEAD; ++x) {
            if (c0 + x < chunks) {
                const float4 d = sum[x];
                const float f = w[x];
                ask(c0 + x + WC_AHEAD, x);
                *reinterpret_cast<float4*>(unit + (c0 + x) * step + e) = s;
                s = make_float4(fmaf(f, s.x, d.x), fmaf(f, s.y, d.y), fmaf(f, s.z, d.z), fmaf(f, s.w, d.w));
            }
        }
    }
    *reinterpret_cast<float4*>(st) = s;
    if (head == 0) {        // the last row's h, for the token shift of the sequence's next token
        float* last = a.state + (int64_t)slot * a.state_stride + (int64_t)a.heads * WC_N * WC_N;
        const bf16* hr = a.h + (int64_t)(row0 + rows - 1) * a.width;
        for (int x = blockIdx.z * WC_STATE_THREADS + threadIdx.x; x < a.width; x += gridDim.z * WC_STATE_THREADS) last[x] = to_f32(hr[x]);
    }
}

struct WkvChunkShared {
    union {
        struct {
            float w[WC_L][WC_N];                   // decays
            bf16 r[WC_L][WC_N + 32], k[WC_L][WC_N + 32];
            float kd[WC_L][WC_PITCH_ROW];          // k times the decays of its block's later tokens
        } in;
        struct {
            float v[WC_L][WC_PITCH_COL];
            uint32_t s[2][WC_N][WC_PITCH_COL];     // the state's two TF32 numbers
        } of;
    };
    float rd[WC_L][WC_PITCH_ROW];                  // r times the decays of its block's earlier tokens
    float A[WC_L][WC_PITCH_ROW];
    float block_decay[WC_BLOCKS][WC_N], before[WC_BLOCKS][WC_N];      // a block's decays; those of all earlier blocks
    float u[WC_N];
};

__device__ __forceinline__ void wc_load4(const bf16* p, float (&x)[4]) {
    const uint2 q = *reinterpret_cast<const uint2*>(p);
    x[0] = __uint_as_float(q.x << 16); x[1] = __uint_as_float(q.x & 0xffff0000u);
    x[2] = __uint_as_float(q.y << 16); x[3] = __uint_as_float(q.y & 0xffff0000u);
}

__global__ void __launch_bounds__(WC_THREADS, 2) wkv_chunk_out_kernel(WkvChunkArgs a) {
    extern __shared__ __align__(16) unsigned char wc_smem[];
    WkvChunkShared& sh = *reinterpret_cast<WkvChunkShared*>(wc_smem);
    pdl_launch_dependents();
    const int tid = threadIdx.x, c = blockIdx.x, seq = blockIdx.y, head = blockIdx.z;
    const int row0 = a.seq_first_row[seq], t0 = row0 + c * WC_L, nt = min(WC_L, a.seq_first_row[seq + 1] - t0);
    if (a.seq_slot[seq] < 0 || nt <= 0) return;
    const int64_t ld = (int64_t)a.heads * WC_N, base = (int64_t)t0 * ld + (int64_t)head * WC_N;
    const int vrow = tid / 8, vcol = tid % 8 * 8;
    uint4 vals = make_uint4(0, 0, 0, 0);           // what the last part needs, on its way from the start
    float4 st[2];
    float odd = 0.f;                               // NaN once a value is not finite
    bool plain;
    {
        const int i = tid % WC_N, b = tid / WC_N;
        const float w0 = a.w0[head * WC_N + i];
        if (b == 0) sh.u[i] = a.u[head * WC_N + i];
        pdl_wait();
        float w[WC_B], r[WC_B], k[WC_B];
#pragma unroll
        for (int x = 0; x < WC_B; ++x) {
            const int t = b * WC_B + x;
            const int64_t at = base + (int64_t)(t < nt ? t : 0) * ld + i;
            w[x] = a.z[at];
            r[x] = to_f32(a.r[at]);
            k[x] = to_f32(a.k[at]);
        }
        if (vrow < nt) vals = *reinterpret_cast<const uint4*>(a.v + base + (int64_t)vrow * ld + vcol);
        const float* unit = wc_unit(a, seq, row0, c, head);
#pragma unroll
        for (int x = 0; x < 2; ++x) st[x] = *reinterpret_cast<const float4*>(unit + 4 * (tid + x * WC_THREADS));
        float all = 1.f;
#pragma unroll
        for (int x = 0; x < WC_B; ++x) {
            const int t = b * WC_B + x;
            w[x] = t < nt ? wc_decay(w[x], w0) : 1.f;
            if (t >= nt) r[x] = k[x] = 0.f;
            odd = fmaf(r[x], 0.f, fmaf(k[x], 0.f, fmaf(w[x], 0.f, odd)));
            sh.in.w[t][i] = w[x];
            sh.in.r[t][i] = __float2bfloat16_rn(r[x]);         // (exact: they came as bfloat16)
            sh.in.k[t][i] = __float2bfloat16_rn(k[x]);
            sh.rd[t][i] = r[x] * all;
            all *= w[x];
        }
        sh.block_decay[b][i] = all;
        float later = 1.f;
#pragma unroll
        for (int x = WC_B - 1; x >= 0; --x) {
            sh.in.kd[b * WC_B + x][i] = k[x] * later;
            later *= w[x];
        }
        plain = __syncthreads_and(odd == 0.f);
        float earlier = 1.f;
#pragma unroll
        for (int x = 0; x < WC_BLOCKS - 1; ++x)
            if (x < b) earlier *= sh.block_decay[x][i];
        sh.before[b][i] = earlier;
    }
    const int lane = tid & 31, warp = tid >> 5, g = lane >> 2, t = lane & 3;
    // A inside a block: eight lanes share a source token s (eight channels each) and walk the targets behind it
    {
        const int b0 = (warp >> 1) * WC_B, s = 4 * (warp & 1) + (lane >> 3), e = lane & 7, row = b0 + s;
        float x[2][4], sum = 0.f;
#pragma unroll
        for (int y = 0; y < 2; ++y) {
            float r4[4];
            wc_load4(&sh.in.k[row][32 * y + 4 * e], x[y]);
            wc_load4(&sh.in.r[row][32 * y + 4 * e], r4);
#pragma unroll
            for (int d = 0; d < 4; ++d) sum = fmaf(r4[d], sh.u[32 * y + 4 * e + d] * x[y][d], sum);
        }
        sum += __shfl_xor_sync(0xffffffffu, sum, 1);
        sum += __shfl_xor_sync(0xffffffffu, sum, 2);
        sum += __shfl_xor_sync(0xffffffffu, sum, 4);
        if (e == 0) sh.A[row][row] = sum;
        if (e < s) sh.A[b0 + e][row] = 0.f;
        if (((warp >> 1) & 1) != 0) sh.A[b0 - WC_B + e][row] = 0.f;          // (the tiles of 16 tokens that the last product takes)
#pragma unroll
        for (int m = 1; m < WC_B; ++m) {
            const int target = min(row + m, b0 + WC_B - 1);
            sum = 0.f;
#pragma unroll
            for (int y = 0; y < 2; ++y) {
                float r4[4];
                wc_load4(&sh.in.r[target][32 * y + 4 * e], r4);
                const float4 w4 = *reinterpret_cast<const float4*>(&sh.in.w[target][32 * y + 4 * e]);
                const float ww[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
                for (int d = 0; d < 4; ++d) {
                    sum = fmaf(r4[d], x[y][d], sum);
                    x[y][d] *= ww[d];
                }
            }
            sum += __shfl_xor_sync(0xffffffffu, sum, 1);
            sum += __shfl_xor_sync(0xffffffffu, sum, 2);
            sum += __shfl_xor_sync(0xffffffffu, sum, 4);
            if (e == 0 && s + m < WC_B) sh.A[row + m][row] = sum;
        }
    }
    // A between blocks: a warp takes a tile of 16 targets (blocks 2 m, 2 m + 1) and the 8 sources of one block sb <= 2 m
    {
        const int m = warp < 1 ? 0 : warp < 4 ? 1 : warp < 9 ? 2 : 3, sb = warp - m * m;
        float sum[1][4] = {}, acc[1][4] = {}, low[1][4] = {};
        if (!plain) {
#pragma unroll 1
            for (int i = 0; i < WC_N; ++i) {
                float f0 = 1.f;
#pragma unroll 1
                for (int b = sb + 1; b < 2 * m; ++b) f0 *= sh.block_decay[b][i];
                const float f1 = sb < 2 * m ? f0 * sh.block_decay[2 * m][i] : 1.f;
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[0][e] = fmaf(sh.rd[16 * m + g + 8 * (e >> 1)][i] * (e >= 2 ? f1 : f0), sh.in.kd[sb * WC_B + 2 * t + (e & 1)][i], sum[0][e]);
            }
        } else
#pragma unroll
        for (int i = 0; i < WC_N; i += 8) {
            float f[2][2];                                      // [place][half of the targets]: the blocks between
#pragma unroll
            for (int p = 0; p < 2; ++p) {
                f[p][0] = 1.f;
                for (int b = sb + 1; b < 2 * m; ++b) f[p][0] *= sh.block_decay[b][i + t + 4 * p];
                f[p][1] = sb < 2 * m ? f[p][0] * sh.block_decay[2 * m][i + t + 4 * p] : 1.f;
            }
            uint32_t hi[4], lo[4], bh[2], bl[2];
#pragma unroll
            for (int e = 0; e < 4; ++e) wc_split(sh.rd[16 * m + g + 8 * (e & 1)][i + t + 4 * (e >> 1)] * f[e >> 1][e & 1], hi[e], lo[e]);
#pragma unroll
            for (int e = 0; e < 2; ++e) wc_split(sh.in.kd[sb * WC_B + g][i + t + 4 * e], bh[e], bl[e]);
            wc_mma(acc[0], hi, bh);
            wc_mma(low[0], hi, bl);
            wc_mma(low[0], lo, bh);
            if (i % 16 == 8) wc_add(sum, acc, low);
        }
#pragma unroll
        for (int e = 0; e < 4; ++e)
            if (e >= 2 || sb < 2 * m) sh.A[16 * m + g + 8 * (e >> 1)][sb * WC_B + 2 * t + (e & 1)] = sum[0][e];
    }
    // values and state take the place of what A was made of
    const float value[8] = {__uint_as_float(vals.x << 16), __uint_as_float(vals.x & 0xffff0000u), __uint_as_float(vals.y << 16), __uint_as_float(vals.y & 0xffff0000u),
                            __uint_as_float(vals.z << 16), __uint_as_float(vals.z & 0xffff0000u), __uint_as_float(vals.w << 16), __uint_as_float(vals.w & 0xffff0000u)};
    const float from[8] = {st[0].x, st[0].y, st[0].z, st[0].w, st[1].x, st[1].y, st[1].z, st[1].w};
#pragma unroll
    for (int e = 0; e < 8; ++e) odd = fmaf(value[e], 0.f, fmaf(from[e], 0.f, odd));
    plain = __syncthreads_and(odd == 0.f);
#pragma unroll
    for (int e = 0; e < 8; e += 2) *reinterpret_cast<float2*>(&sh.of.v[vrow][vcol + e]) = make_float2(value[e], value[e + 1]);
#pragma unroll
    for (int x = 0; x < 2; ++x) {
        const int at = tid + x * WC_THREADS;
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            wc_split(from[4 * x + e], hi[e], lo[e]);
            if (!plain) hi[e] = __float_as_uint(from[4 * x + e]);
        }
        *reinterpret_cast<uint4*>(&sh.of.s[0][at / (WC_N / 4)][at % (WC_N / 4) * 4]) = make_uint4(hi[0], hi[1], hi[2], hi[3]);
        *reinterpret_cast<uint4*>(&sh.of.s[1][at / (WC_N / 4)][at % (WC_N / 4) * 4]) = make_uint4(lo[0], lo[1], lo[2], lo[3]);
    }
    __syncthreads();
    const int m = warp & 3, j0 = 16 * (warp >> 2);
    float sum[2][4] = {}, acc[2][4] = {}, low[2][4] = {};
    if (plain)
#pragma unroll
    for (int i = 0; i < WC_N; i += 8) {
        uint32_t hi[4], lo[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) wc_split(sh.rd[16 * m + g + 8 * (e & 1)][i + t + 4 * (e >> 1)] * sh.before[2 * m + (e & 1)][i + t + 4 * (e >> 1)], hi[e], lo[e]);
#pragma unroll
        for (int n = 0; n < 2; ++n) {
            const uint32_t bh[2] = {sh.of.s[0][i + t][j0 + 8 * n + g], sh.of.s[0][i + t + 4][j0 + 8 * n + g]};
            const uint32_t bl[2] = {sh.of.s[1][i + t][j0 + 8 * n + g], sh.of.s[1][i + t + 4][j0 + 8 * n + g]};
            wc_mma(acc[n], hi, bh);
            wc_mma(low[n], hi, bl);
            wc_mma(low[n], lo, bh);
        }
        if (i % 16 == 8) wc_add(sum, acc, low);
    }
    if (plain) {
        for (int s0 = 0; s0 <= m * 16; s0 += 16) {
#pragma unroll
            for (int s = s0; s < s0 + 16; s += 8) {
                uint32_t hi[4], lo[4];
#pragma unroll
                for (int e = 0; e < 4; ++e) wc_split(sh.A[16 * m + g + 8 * (e & 1)][s + t + 4 * (e >> 1)], hi[e], lo[e]);
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const uint32_t bv[2] = {__float_as_uint(sh.of.v[s + t][j0 + 8 * n + g]), __float_as_uint(sh.of.v[s + t + 4][j0 + 8 * n + g])};
                    wc_mma(acc[n], hi, bv);
                    wc_mma(low[n], lo, bv);
                }
            }
            wc_add(sum, acc, low);
        }
    } else {                // (nor may a value that is not finite meet the zeros of the tokens before it)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int target = 16 * m + g + 8 * (e >> 1), j = j0 + 8 * n + 2 * t + (e & 1);
#pragma unroll 1
                for (int i = 0; i < WC_N; ++i)
                    sum[n][e] = fmaf(sh.rd[target][i] * sh.before[2 * m + (e >> 1)][i], __uint_as_float(sh.of.s[0][i][j]), sum[n][e]);
#pragma unroll 1
                for (int s = 0; s <= target; ++s) sum[n][e] = fmaf(sh.A[target][s], sh.of.v[s][j], sum[n][e]);
            }
    }
#pragma unroll
    for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int e = 0; e < 2; ++e) {
            const int target = 16 * m + g + 8 * e;
            if (target < nt) *reinterpret_cast<float2*>(a.o + base + (int64_t)target * ld + j0 + 8 * n + 2 * t) = make_float2(sum[n][2 * e], sum[n][2 * e + 1]);
        }
}

X0NE_API int x0ne_wkv_chunk_tokens() { return WC_L; }
X0NE_API int x0ne_wkv_chunk_unit() { return WC_UNIT; }

// bfloat16 runs of heads of 64; at most max_seq_rows rows per sequence; scratch: (n_rows / 64 + n_seqs) x heads x WC_UNIT floats.  The rest as for
// x0ne_wkv_scan.
X0NE_API int x0ne_wkv_chunk_scan(const void* r, const void* k, const void* v, const float* z, const float* w0, const float* u, const void* h, float* o, float* state,
                                 int64_t state_stride, const int32_t* seq_first_row, const int32_t* seq_slot, int n_seqs, int n_rows, int max_seq_rows, int heads, int width,
                                 float* scratch, int64_t scratch_floats, cudaStream_t stream) {
    X0NE_REQUIRE(n_seqs >= 0 && n_seqs <= 65535 && n_rows >= 0 && max_seq_rows >= 0 && heads > 0 && heads <= 65535 && width > 0 &&
                     state_stride >= (int64_t)heads * WC_N * WC_N + width && state_stride % 4 == 0,
                 "wkv_chunk_scan: %d sequences, %d heads, width %d", n_seqs, heads, width);
    X0NE_REQUIRE(scratch != nullptr && scratch_floats >= ((int64_t)n_rows / WC_L + n_seqs) * heads * WC_UNIT, "wkv_chunk_scan: %lld floats of scratch", (long long)scratch_floats);
    X0NE_REQUIRE((((uintptr_t)v | (uintptr_t)o | (uintptr_t)state | (uintptr_t)scratch) & 15) == 0, "wkv_chunk_scan: a tensor is not 16-byte aligned");
    if (n_seqs == 0 || max_seq_rows == 0) return 0;
    WkvChunkArgs a{(const bf16*)r, (const bf16*)k, (const bf16*)v, z, w0, u, (const bf16*)h, o, state, scratch, state_stride, seq_first_row, seq_slot, heads, width};
    static OncePerDevice configured;
    if (configured.need()) {
        const cudaError_t e = cudaFuncSetAttribute(wkv_chunk_out_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(WkvChunkShared));
        X0NE_REQUIRE(e == cudaSuccess, "wkv_chunk_scan: %zu bytes of shared memory: %s", sizeof(WkvChunkShared), cudaGetErrorString(e));
        configured.done();
    }
    const dim3 grid((max_seq_rows + WC_L - 1) / WC_L, n_seqs, heads);
    x0ne_launch(wkv_chunk_sums_kernel, grid, dim3(WC_THREADS), 0, stream, a);
    cudaError_t e = cudaGetLastError();
    X0NE_REQUIRE(e == cudaSuccess, "wkv_chunk_scan: %s", cudaGetErrorString(e));
    x0ne_launch(wkv_chunk_states_kernel, dim3(n_seqs, heads, WC_N * WC_N / 4 / WC_STATE_THREADS), dim3(WC_STATE_THREADS), 0, stream, a);
    e = cudaGetLastError();
    X0NE_REQUIRE(e == cudaSuccess, "wkv_chunk_scan: %s", cudaGetErrorString(e));
    x0ne_launch(wkv_chunk_out_kernel, grid, dim3(WC_THREADS), sizeof(WkvChunkShared), stream, a);
    X0NE_LAUNCH_CHECK();
}
