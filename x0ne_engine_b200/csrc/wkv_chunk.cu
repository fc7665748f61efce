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
// logarithms: nothing overflows, a factor that underflows belongs to a term that does.  Inside a block of 8 tokens A is made by multiply-adds over
// running products; A between blocks and the outputs are products of matrices on mma.sync m16n8k16 with every float32 operand as three bfloat16
// numbers, which hold all of it (v is exact as one), the products of the largest parts in an accumulator of their own, added up in float32 every
// 16 terms.  The tensor core cuts its sums off, so what is most of a result where decays are fast stays with multiply-adds: a chunk's own state is
// walked, an output's own tile of 16 tokens added term by term.  States, decays and sums are float32, products of a whole block's decays are taken in
// 64 bits and rounded once.  The order of sums differs from the token-by-token kernels', which stay for 32-bit runs, steps and short runs.
// Infinities and NaN have no parts (a NaN can even lose itself in the rounding): where a chunk of a head meets one, its products are
// made by multiply-adds of the whole values instead, so that it reaches what it reaches in the token-by-token kernel.
// Error against 64 bits (2-norm over 2-norm; w0 a decay rate, mean of three seeds), outputs and states, walk -> here: one chunk, rate 1 7.8e-8 / 3.9e-8 -> 7.4e-8 /
// 3.6e-8, rate 0.01 1.67e-7 / 1.90e-7 -> 1.63e-7 / 1.85e-7; four sequences of 128, rate 0.1 1.06e-7 / 8.7e-8 -> 1.06e-7 / 8.4e-8; 2,048 tokens, rate 0.01 2.31e-7 / 2.25e-7 ->
// 2.17e-7 / 2.10e-7.  With two TF32 numbers to an operand and everything on the tensor core it was 9.5e-8 / 6.4e-8 in the first of these, 2.49e-7 / 2.24e-7 in the last.
// The scan of one sequence of 2,048 tokens, 32 heads: 146 -> 107 us (91 in that other form), 16 heads 146 -> 68, 64 heads 251 -> 206; 16 sequences of 128, 32 heads
// 124 -> 103.
#include "common.cuh"

#define WC_L 64                 // tokens of a chunk
#define WC_B 8                  // tokens of a block
#define WC_BLOCKS (WC_L / WC_B)
#define WC_N 64                 // channels of a head
#define WC_THREADS 512
#define WC_STATE_THREADS 256
#define WC_PITCH_ROW 72         // floats between rows that fragments read along (4 rows x 4 pairs meet 32 banks)
#define WC_PITCH_COL 68         // and across (every second row of 4, 8 places)
#define WC_PITCH_PAIR 72        // and of rows of pairs (4 rows x 8 places)
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
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3]) : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// two values as three bfloat16 each, exactly: x rounded, what is left of it rounded, and the rest (x in the lower halves)
__device__ __forceinline__ void wc_split(float x, float y, uint32_t& a, uint32_t& b, uint32_t& c) {
    auto pack = [&](uint32_t& to) { asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(to) : "f"(y), "f"(x)); };
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
// two float32 numbers that are bfloat16 numbers
__device__ __forceinline__ uint32_t wc_pair(float x, float y) { return __byte_perm(__float_as_uint(x), __float_as_uint(y), 0x7632); }
__device__ __forceinline__ float wc_decay(float z, float w0) { return expf(-expf(z + w0)); }
// where chunk c of a sequence that starts at row0 keeps its scratch (a sequence of n rows has ceil(n / 64) chunks, so no two meet)
__device__ __forceinline__ float* wc_unit(const WkvChunkArgs& a, int seq, int row0, int c, int head) {
    return a.scratch + ((int64_t)(row0 / WC_L + seq + c) * a.heads + head) * WC_UNIT;
}

#define WC_CAREFUL 4            // tokens at a chunk's end whose roundings are made up for
// B and the product of decays.  A thread takes one channel of one block of tokens, then four key channels x two value channels, which it walks from zero
// as the token-by-token kernel walks them: products of matrices were 12 us faster for 2,048 tokens of 32 heads, but the tensor core cuts its sums off, and
// a state that forgets fast came out 6.1e-8 off 64 bits instead of 3.9e-8 (multiply-adds of k times its later decays: 2.1e-7 instead of 1.9e-7 for a slow one).
__global__ void __launch_bounds__(WC_THREADS, 3) wkv_chunk_sums_kernel(WkvChunkArgs a) {
    __shared__ __align__(16) float ws[WC_L][WC_N], ks[WC_L][WC_N], vs[WC_L][WC_N];
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
    double all = 1.;                    // (64 bits: the decays of a whole chunk in one number would be 64 roundings off otherwise)
#pragma unroll
    for (int x = 0; x < WC_B; ++x) {
        const int t = b * WC_B + x;
        if (t >= nt) continue;
        const float d = wc_decay(w[x], w0);
        ws[t][i] = d;
        ks[t][i] = k[x];
        vs[t][i] = v[x];
        all *= d;
    }
    __syncthreads();
    const int lane = tid & 31, warp = tid >> 5;
    float2 sum[4] = {};
    const int last = max(0, nt - WC_CAREFUL);
#pragma unroll 4
    for (int t = 0; t < last; ++t) {
        const float4 d = *reinterpret_cast<const float4*>(&ws[t][4 * warp]), x = *reinterpret_cast<const float4*>(&ks[t][4 * warp]);
        const float2 y = *reinterpret_cast<const float2*>(&vs[t][2 * lane]);
        sum[0] = __ffma2_rn(make_float2(d.x, d.x), sum[0], __fmul2_rn(make_float2(x.x, x.x), y));
        sum[1] = __ffma2_rn(make_float2(d.y, d.y), sum[1], __fmul2_rn(make_float2(x.y, x.y), y));
        sum[2] = __ffma2_rn(make_float2(d.z, d.z), sum[2], __fmul2_rn(make_float2(x.z, x.z), y));
        sum[3] = __ffma2_rn(make_float2(d.w, d.w), sum[3], __fmul2_rn(make_float2(x.w, x.w), y));
    }
    // the newest tokens with what each rounding leaves (k v is exact), so that the rounding of B itself and the one behind it are no more than a
    // walk's (5 us of 2,048 tokens of 32 heads; without it states of 100 to 128 tokens were 4 to 5 % further off than the walk's)
    float2 rest[4] = {};
#pragma unroll 1
    for (int t = last; t < nt; ++t) {
        const float2 y = *reinterpret_cast<const float2*>(&vs[t][2 * lane]);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float d1 = ws[t][4 * warp + e], x1 = ks[t][4 * warp + e];
            const float2 d = make_float2(d1, d1), add = __fmul2_rn(make_float2(x1, x1), y), p = __fmul2_rn(d, sum[e]);
            const float2 left = __ffma2_rn(d, sum[e], make_float2(-p.x, -p.y)), s = __fadd2_rn(p, add), b2 = __fadd2_rn(s, make_float2(-p.x, -p.y));
            const float2 a2 = __fadd2_rn(s, make_float2(-b2.x, -b2.y));
            const float2 off = __fadd2_rn(__fadd2_rn(p, make_float2(-a2.x, -a2.y)), __fadd2_rn(add, make_float2(-b2.x, -b2.y)));
            rest[e] = __ffma2_rn(d, rest[e], __fadd2_rn(left, off));
            sum[e] = s;
        }
    }
#pragma unroll
    for (int e = 0; e < 4; ++e) {
        const float2 s = __fadd2_rn(sum[e], rest[e]);
        sum[e] = make_float2(fabsf(sum[e].x) < INFINITY ? s.x : sum[e].x, fabsf(sum[e].y) < INFINITY ? s.y : sum[e].y);       // (an infinity leaves NaN)
    }
    float* unit = wc_unit(a, seq, row0, c, head);
#pragma unroll
    for (int e = 0; e < 4; ++e) *reinterpret_cast<float2*>(unit + (4 * warp + e) * WC_N + 2 * lane) = sum[e];
    __syncthreads();
    double (*of_block)[WC_N] = reinterpret_cast<double (*)[WC_N]>(&ws[0][0]);
    of_block[b][i] = all;
    __syncthreads();
    if (b == 0) {
#pragma unroll
        for (int x = 1; x < WC_BLOCKS; ++x) all *= of_block[x][i];
        unit[WC_N * WC_N + i] = (float)all;
    }
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

// Sums of products stay in the tensor core for 16 terms and are added up with rounding from there on (it cuts its sums off); the products of
// the largest parts have an accumulator of their own.
template <int NT>
__device__ __forceinline__ void wc_add(float (&sum)[NT][4], float (&acc)[NT][4], float (&low)[NT][4]) {
#pragma unroll
    for (int n = 0; n < NT; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            sum[n][e] = (sum[n][e] + low[n][e]) + acc[n][e];
            acc[n][e] = low[n][e] = 0.f;
        }
}

// a x b from both operands' three parts, the smallest products first
__device__ __forceinline__ void wc_products(float (&acc)[4], float (&low)[4], const uint32_t (&a)[3][4], const uint32_t (&b0)[2], const uint32_t (&b1)[2], const uint32_t (&b2)[2]) {
    wc_mma(acc, a[0], b0);
    wc_mma(low, a[1], b2);
    wc_mma(low, a[2], b1);
    wc_mma(low, a[0], b2);
    wc_mma(low, a[1], b1);
    wc_mma(low, a[2], b0);
    wc_mma(low, a[0], b1);
    wc_mma(low, a[1], b0);
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
            union {
                uint32_t s[3][WC_N / 2][WC_PITCH_PAIR];        // the state's three bfloat16 numbers, two key channels together
                float whole[WC_N][WC_PITCH_PAIR];              // (as it is, where something is not finite)
            };
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
        for (int x = 0; x < 2; ++x) st[x] = *reinterpret_cast<const float4*>(unit + (tid / 16 * 2 + x) * WC_N + tid % 16 * 4);
        float all = 1.f;
        double block = 1.;
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
            block *= w[x];
        }
        sh.block_decay[b][i] = (float)block;
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
        for (int i = 0; i < WC_N; i += 16) {
            uint32_t a3[3][4], b3[3][2];
#pragma unroll
            for (int p = 0; p < 2; ++p) {                       // [place][half of the targets]: times the blocks between
                const int at = i + 2 * t + 8 * p;
                float2 f = make_float2(1.f, 1.f);
                for (int b = sb + 1; b < 2 * m; ++b) {
                    const float2 d = *reinterpret_cast<const float2*>(&sh.block_decay[b][at]);
                    f.x *= d.x;
                    f.y *= d.y;
                }
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float2 r = *reinterpret_cast<const float2*>(&sh.rd[16 * m + g + 8 * half][at]);
                    wc_split(r.x * f.x, r.y * f.y, a3[0][2 * p + half], a3[1][2 * p + half], a3[2][2 * p + half]);
                    if (half == 0 && sb < 2 * m) {
                        const float2 d = *reinterpret_cast<const float2*>(&sh.block_decay[2 * m][at]);
                        f.x *= d.x;
                        f.y *= d.y;
                    }
                }
                const float2 k = *reinterpret_cast<const float2*>(&sh.in.kd[sb * WC_B + g][at]);
                wc_split(k.x, k.y, b3[0][p], b3[1][p], b3[2][p]);
            }
            wc_products(acc[0], low[0], a3, b3[0], b3[1], b3[2]);
            wc_add(sum, acc, low);
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
    const int q = tid / 16, qcol = tid % 16 * 4;           // its key channels 2 q and 2 q + 1
    if (plain) {
        uint32_t p[3][4];
#pragma unroll
        for (int e = 0; e < 4; ++e) wc_split(from[e], from[4 + e], p[0][e], p[1][e], p[2][e]);
#pragma unroll
        for (int o = 0; o < 3; ++o) *reinterpret_cast<uint4*>(&sh.of.s[o][q][qcol]) = make_uint4(p[o][0], p[o][1], p[o][2], p[o][3]);
    } else {
#pragma unroll
        for (int x = 0; x < 2; ++x) *reinterpret_cast<float4*>(&sh.of.whole[2 * q + x][qcol]) = st[x];
    }
    __syncthreads();
    const int m = warp & 3, j0 = 16 * (warp >> 2);
    float sum[2][4] = {}, acc[2][4] = {}, low[2][4] = {};
    if (plain) {
#pragma unroll
        for (int i = 0; i < WC_N; i += 16) {
            uint32_t a3[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int at = i + 2 * t + 8 * (e >> 1);
                const float2 r = *reinterpret_cast<const float2*>(&sh.rd[16 * m + g + 8 * (e & 1)][at]), d = *reinterpret_cast<const float2*>(&sh.before[2 * m + (e & 1)][at]);
                wc_split(r.x * d.x, r.y * d.y, a3[0][e], a3[1][e], a3[2][e]);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                uint32_t b3[3][2];
#pragma unroll
                for (int p = 0; p < 3; ++p)
#pragma unroll
                    for (int e = 0; e < 2; ++e) b3[p][e] = sh.of.s[p][i / 2 + t + 4 * e][j0 + 8 * n + g];
                wc_products(acc[n], low[n], a3, b3[0], b3[1], b3[2]);
            }
            wc_add(sum, acc, low);
        }
        for (int s = 0; s < m * 16; s += 16) {
            uint32_t a3[3][4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 x = *reinterpret_cast<const float2*>(&sh.A[16 * m + g + 8 * (e & 1)][s + 2 * t + 8 * (e >> 1)]);
                wc_split(x.x, x.y, a3[0][e], a3[1][e], a3[2][e]);
            }
#pragma unroll
            for (int n = 0; n < 2; ++n) {
                const int j = j0 + 8 * n + g;
                const uint32_t bv[2] = {wc_pair(sh.of.v[s + 2 * t][j], sh.of.v[s + 2 * t + 1][j]), wc_pair(sh.of.v[s + 2 * t + 8][j], sh.of.v[s + 2 * t + 9][j])};
                wc_mma(acc[n], a3[0], bv);
                wc_mma(low[n], a3[2], bv);
                wc_mma(low[n], a3[1], bv);
            }
            wc_add(sum, acc, low);
        }
        // the target's own tile of 16 tokens by multiply-adds: the newest tokens are most of an output where decays are fast
#pragma unroll
        for (int s = 16 * m; s < 16 * m + 16; s += 4) {
            float a4[2][4];
#pragma unroll
            for (int e = 0; e < 2; ++e) *reinterpret_cast<float4*>(a4[e]) = *reinterpret_cast<const float4*>(&sh.A[16 * m + g + 8 * e][s]);
#pragma unroll
            for (int x = 0; x < 4; ++x)
#pragma unroll
                for (int n = 0; n < 2; ++n) {
                    const float2 y = *reinterpret_cast<const float2*>(&sh.of.v[s + x][j0 + 8 * n + 2 * t]);
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const float2 o = __ffma2_rn(make_float2(a4[e][x], a4[e][x]), y, make_float2(sum[n][2 * e], sum[n][2 * e + 1]));
                        sum[n][2 * e] = o.x;
                        sum[n][2 * e + 1] = o.y;
                    }
                }
        }
    } else {                // (nor may a value that is not finite meet the zeros of the tokens before it)
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int target = 16 * m + g + 8 * (e >> 1), j = j0 + 8 * n + 2 * t + (e & 1);
#pragma unroll 1
                for (int i = 0; i < WC_N; ++i)
                    sum[n][e] = fmaf(sh.rd[target][i] * sh.before[2 * m + (e >> 1)][i], sh.of.whole[i][j], sum[n][e]);
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
