// The delta rule and the generalized one (recurrent.cu) for rows of many tokens, eight tokens a step, everything in 32-bit on CUDA
// cores, for key sizes of 64, 128 and 256.
//
// Token by token a scan is a chain: decay, a sum over the key channels' lanes, the write, the next token (2,048 tokens of 16
// heads of 128 by 128 with the delta rule: 568 us, 278 ns a token). Over a block of T = 8 tokens with the state S before it, the
// inputs' decayed products and the sums that involve S alone need no such chain. With G_j = g_1 o .. o g_j (per key channel)
// and j, i counting the block's tokens,
//     o_j = S^T (G_j o q_j) + sum_(i <= j) N_ji u_i,           N_ji = q_j . (g_(i+1) o .. o g_j o k_i)
//     S'  = G_T o S + sum_i k'_i u_i^T,                        k'_i = g_(i+1) o .. o g_T o k_i
// with (u_j = beta_j (v_j - S_j-^T k_j), S_j- the state decayed for token j)
//     u_j = beta_j (d_j - sum_(i < j) M_ji u_i),   d_j = v_j - S^T (G_j o k_j),   M_ji = k_j . (g_(i+1) o .. o g_j o k_i),
// a triangular system that S has no part in: u = A d, so with N A for N and sum_j k'_j A_ji for k'_i the block needs d alone
// (the form of Bischof and Van Loan for products of Householder matrices, here with decays). The generalized rule (S_j = g_j o S_(j-1) +
// k_j v_j^T - (r_j o k_j) a_j^T, a_j = S_(j-1)^T k_j) gives such sums over v and over x_j = S^T (G_(j-1) o k_j). Products of
// decays only, never quotients: a decay of zero is nothing special. G is kept as a sum of two floats and G_T applied as one:
// with a fixed decay its rounding would be the same in every block and add up over the blocks that S remembers. The block's
// writes are summed before they meet S, which then rounds once a block. A token that is no finite number reaches no earlier one.
//   recurrent_block_kernel    a warp per (block, head): the decayed vectors and N, which all columns of S share, to scratch.
//   recurrent_blocks_kernel   a CTA per (row, head, 16 columns of S) walks the row's blocks with its columns in registers: a
//                             thread holds 8 (4) channels of two or four columns, so that a vector's 16 bytes from shared memory meet as
//                             many numbers of S; sums over the 16 (32) lanes of a column by halving the values a lane still
//                             holds, 15 shuffles for 16 sums; packed multiply-adds; blocks arrive by cp.async, two ahead.
// Bound by the issue of its instructions, about 1,200 a block for a warp of eight columns, at one warp a scheduler. 305 us at the size above.
#include "common.cuh"

#define RB_T 8
#define RB_STAGES 3
#define RB_VT 16                                          // columns a CTA
enum { RB_DELTA = 1, RB_GENERAL = 2 };

// What the first kernel leaves for a (block, head), in floats: [G_j o k_j] [G_j o q_j] [what d (RB_GENERAL: v) writes]
// [what -x writes (RB_GENERAL)], each [T][dim]; G_T [dim] and what its rounding lost [dim]; the read-outs' shares N of the
// writes [T][T], twice for RB_GENERAL.
static __host__ __device__ constexpr int rb_vectors(int mode) { return mode == RB_DELTA ? 3 : 4; }
static __host__ __device__ constexpr int rb_floats(int mode, int dim) {
    return rb_vectors(mode) * RB_T * dim + 2 * dim + (mode == RB_GENERAL ? 2 : 1) * RB_T * RB_T;
}

__device__ __forceinline__ void rb_fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t rb_twice(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float rb_sum(uint64_t v) {
    float a, b;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
    return a + b;
}

// Sums of V values over P neighbouring lanes (V <= P, powers of two): lane p leaves with the sum of value p mod V.
template <int V, int P>
__device__ __forceinline__ float lanes_sum(float (&x)[V], int p) {
#pragma unroll
    for (int o = V / 2; o > 0; o >>= 1) {
        const bool up = p & o;
#pragma unroll
        for (int i = 0; i < o; ++i) {
            const float send = up ? x[i] : x[i + o], keep = up ? x[i + o] : x[i];
            x[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
        }
    }
#pragma unroll
    for (int o = V; o < P; o <<= 1) x[0] += __shfl_xor_sync(0xffffffffu, x[0], o);
    return x[0];
}

template <int C> struct Channels { float x[C]; };        // a lane's C neighbouring channels
template <int C>
__device__ __forceinline__ Channels<C> rb_load(const float* p) {
    Channels<C> r;
    if constexpr (C == 2) { const float2 v = *(const float2*)p; r.x[0] = v.x; r.x[1] = v.y; }
    else {
#pragma unroll
        for (int i = 0; i < C; i += 4) { const float4 v = *(const float4*)(p + i); r.x[i] = v.x; r.x[i + 1] = v.y; r.x[i + 2] = v.z; r.x[i + 3] = v.w; }
    }
    return r;
}
template <int C>
__device__ __forceinline__ void rb_store(float* p, const Channels<C>& r) {
    if constexpr (C == 2) *(float2*)p = make_float2(r.x[0], r.x[1]);
    else {
#pragma unroll
        for (int i = 0; i < C; i += 4) *(float4*)(p + i) = make_float4(r.x[i], r.x[i + 1], r.x[i + 2], r.x[i + 3]);
    }
}
template <int C>
__device__ __forceinline__ Channels<C> rb_all(float f) {
    Channels<C> r;
#pragma unroll
    for (int i = 0; i < C; ++i) r.x[i] = f;
    return r;
}
template <int C>
__device__ __forceinline__ Channels<C> rb_mul(const Channels<C>& a, const Channels<C>& b) {
    Channels<C> r;
#pragma unroll
    for (int i = 0; i < C; ++i) r.x[i] = a.x[i] * b.x[i];
    return r;
}
template <int C>
__device__ __forceinline__ float rb_dot(const Channels<C>& a, const Channels<C>& b) {
    float s = 0.f;
#pragma unroll
    for (int i = 0; i < C; ++i) s = fmaf(a.x[i], b.x[i], s);
    return s;
}

// Blocks of row b: ceil(tokens / 8), and none of a row of fewer than `least` tokens (the token-by-token scan's).
__device__ __forceinline__ int blocks_of(const int32_t* __restrict__ query_start, int b, int least) {
    const int n = query_start[b + 1] - query_start[b];
    return n >= least ? (n + RB_T - 1) / RB_T : 0;
}

// grid (blocks, heads / 4), 128 threads
template <int C, int MODE>
__global__ void __launch_bounds__(128) recurrent_block_kernel(float* __restrict__ scratch, const float* __restrict__ qk,
                                                              const float* __restrict__ decay, const float* __restrict__ head_decay,
                                                              const float* __restrict__ beta, const float* __restrict__ rate,
                                                              const int32_t* __restrict__ query_start, int row0, int rows, int least,
                                                              int heads, int kv_heads) {
    constexpr int DIM = 32 * C;
    __shared__ float products[4][2][RB_T][2 * RB_T], system[4][2][RB_T][RB_T];   // per warp: [N | M] of k, of r o k; A, B
    const int h = blockIdx.y * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (h >= heads) return;
    int left = blockIdx.x, t0 = 0, m = 0;
    for (int b = row0; b < rows; ++b) {
        const int blocks = blocks_of(query_start, b, least);
        if (left < blocks) { t0 = query_start[b] + left * RB_T; m = min(RB_T, query_start[b + 1] - t0); break; }
        left -= blocks;
    }
    if (m == 0) return;                                                  // (more blocks were launched than the step has)
    const int hk = h / (heads / kv_heads);
    float* kd = scratch + ((size_t)blockIdx.x * heads + h) * rb_floats(MODE, DIM) + lane * C;
    float* qd = kd + RB_T * DIM;
    float* kr = qd + RB_T * DIM;
    float* rr = kr + RB_T * DIM;
    float* gT = kr + (MODE == RB_GENERAL ? 2 : 1) * RB_T * DIM;
    float* coef = gT - lane * C + 2 * DIM;
    Channels<C> r[RB_T], s[MODE == RB_GENERAL ? RB_T : 1], G = rb_all<C>(1.f), lost = rb_all<C>(0.f);
    float x[32], y[MODE == RB_GENERAL ? 32 : 1];
#pragma unroll
    for (int j = 0; j < RB_T; ++j) {
        const bool there = j < m;                                        // (what lies past the row: k = q = 0, g = 1, beta = 0)
        const size_t t = t0 + (there ? j : 0);
        const Channels<C> zero = rb_all<C>(0.f);
        const Channels<C> q = there ? rb_load<C>(qk + ((t * 2) * kv_heads + hk) * DIM + lane * C) : zero;
        const Channels<C> k = there ? rb_load<C>(qk + ((t * 2 + 1) * kv_heads + hk) * DIM + lane * C) : zero;
        const Channels<C> g = !there ? rb_all<C>(1.f) : decay ? rb_load<C>(decay + (t * heads + h) * DIM + lane * C) : rb_all<C>(head_decay[h]);
        float* xn = x + (j & 1) * 16;                                    // two tokens' rows [N | M] are summed over the lanes at once
        float* yn = y + (MODE == RB_GENERAL ? (j & 1) * 16 : 0);
        if (MODE == RB_GENERAL) {
#pragma unroll
            for (int i = 0; i < RB_T; ++i) {
                xn[RB_T + i] = i < j ? rb_dot<C>(k, r[i]) : 0.f;
                yn[RB_T + i] = i < j ? rb_dot<C>(k, s[i]) : 0.f;
            }
            rb_store<C>(kd + j * DIM, rb_mul<C>(G, k));
        }
#pragma unroll
        for (int i = 0; i < j; ++i) {
            r[i] = rb_mul<C>(r[i], g);
            if (MODE == RB_GENERAL) s[i] = rb_mul<C>(s[i], g);
        }
#pragma unroll
        for (int i = 0; i < C; ++i) {                                    // (G, lost) *= g
            const float top = G.x[i] * g.x[i], low = fmaf(G.x[i], g.x[i], -top) + lost.x[i] * g.x[i];
            G.x[i] = top + low;
            lost.x[i] = low - (G.x[i] - top);
        }
        if (MODE != RB_GENERAL) {
#pragma unroll
            for (int i = 0; i < RB_T; ++i) xn[RB_T + i] = i < j ? rb_dot<C>(k, r[i]) : 0.f;
            rb_store<C>(kd + j * DIM, rb_mul<C>(G, k));
        }
        r[j] = k;
        if (MODE == RB_GENERAL) s[j] = there ? rb_mul<C>(k, rb_load<C>(rate + (t * heads + h) * DIM + lane * C)) : zero;
#pragma unroll
        for (int i = 0; i < RB_T; ++i) {
            xn[i] = i <= j ? rb_dot<C>(q, r[i]) : 0.f;
            if (MODE == RB_GENERAL) yn[i] = i <= j ? rb_dot<C>(q, s[i]) : 0.f;
        }
        rb_store<C>(qd + j * DIM, rb_mul<C>(G, q));
        if (j & 1) {
            (&products[threadIdx.x >> 5][0][j - 1][0])[lane] = lanes_sum<32, 32>(x, lane);
            if constexpr (MODE == RB_GENERAL) (&products[threadIdx.x >> 5][1][j - 1][0])[lane] = lanes_sum<32, 32>(y, lane);
        }
    }
    rb_store<C>(gT, G);
    rb_store<C>(gT + DIM, lost);
    float (*n)[2 * RB_T] = products[threadIdx.x >> 5][0];
    float (*ns)[2 * RB_T] = products[threadIdx.x >> 5][1];
    float (*A)[RB_T] = system[threadIdx.x >> 5][0];
    float (*B)[RB_T] = system[threadIdx.x >> 5][1];
    __syncwarp();
    if (lane < RB_T) {                                                   // column `lane` of A by forward substitution
        float c[RB_T];
#pragma unroll
        for (int j = 0; j < RB_T; ++j) {
            float sum = j == lane ? 1.f : 0.f;
#pragma unroll
            for (int l = 0; l < j; ++l) sum = l < lane ? sum : fmaf(-(MODE == RB_GENERAL ? ns : n)[j][RB_T + l], c[l], sum);
            c[j] = j < lane ? 0.f : MODE == RB_GENERAL ? sum : j < m ? beta[(size_t)(t0 + j) * heads + h] * sum : 0.f;
            A[j][lane] = c[j];
        }
    }
    __syncwarp();
    if (MODE == RB_GENERAL) {                                            // B = A M: what v has in a
#pragma unroll
        for (int e = lane; e < RB_T * RB_T; e += 32) {
            const int j = e / RB_T, i = e % RB_T;
            float sum = 0.f;
#pragma unroll
            for (int l = 0; l < RB_T; ++l) sum = l <= j && l > i ? fmaf(A[j][l], n[l][RB_T + i], sum) : sum;
            B[j][i] = sum;
        }
        __syncwarp();
    }
#pragma unroll
    for (int e = lane; e < RB_T * RB_T; e += 32) {                       // the read-outs' shares of the writes
        const int j = e / RB_T, i = e % RB_T;
        float sum = 0.f, other = 0.f;
#pragma unroll
        for (int l = 0; l < RB_T; ++l) {
            if (l > j || l < i) continue;                                // (a token that is no number reaches none before it)
            if (MODE == RB_DELTA) sum = fmaf(n[j][l], A[l][i], sum);
            if (MODE == RB_GENERAL) { sum = fmaf(ns[j][l], B[l][i], sum); other = fmaf(ns[j][l], A[l][i], other); }
        }
        coef[e] = MODE == RB_DELTA ? sum : n[j][i] - sum;
        if (MODE == RB_GENERAL) coef[RB_T * RB_T + e] = other;
    }
#pragma unroll
    for (int i = 0; i < RB_T; ++i) {                                     // and what a token's v (d) and x write
        Channels<C> w = MODE == RB_DELTA ? rb_all<C>(0.f) : r[i], z = rb_all<C>(0.f);
#pragma unroll
        for (int j = i; j < RB_T; ++j)
#pragma unroll
            for (int c = 0; c < C; ++c) {
                if (MODE == RB_DELTA) w.x[c] = fmaf(r[j].x[c], A[j][i], w.x[c]);
                if (MODE == RB_GENERAL) {
                    w.x[c] = fmaf(-s[j].x[c], B[j][i], w.x[c]);
                    z.x[c] = fmaf(s[j].x[c], A[j][i], z.x[c]);
                }
            }
        rb_store<C>(kr + i * DIM, w);
        if (MODE == RB_GENERAL) rb_store<C>(rr + i * DIM, z);
    }
}

// grid: rows x column tiles x heads, the heads of a row's tile next to one another (a long row's CTAs are then spread over the chip
// before those of rows that end sooner or are passed over), P * 16 / NC threads: thread (g, p) holds channels (i P + p) 4 .. + 3, i < DPT / 4, of columns
// NC g .. NC g + NC - 1 of the CTA's 16
template <int DPT, int P, int NC, int MODE>
__global__ void __launch_bounds__(P * RB_VT / NC) recurrent_blocks_kernel(
        float* __restrict__ out, const float* __restrict__ scratch, const float* __restrict__ v, float* __restrict__ state,
        const int32_t* __restrict__ query_start, const int32_t* __restrict__ row_slot, int row0, int least, int heads, int vdim) {
    constexpr int DIM = DPT * P, VT = RB_VT, THREADS = P * VT / NC, T = RB_T;
    constexpr int FLOATS = rb_floats(MODE, DIM), STAGE = FLOATS + T * VT, V = 2 * T, QUADS = DPT / 4;
    extern __shared__ float4 smem4[];
    float* sm = (float*)smem4;                                           // [RB_STAGES][STAGE], then the outputs [2][T][VT]
    float* so = sm + RB_STAGES * STAGE;
    const int h = blockIdx.x % heads, part = blockIdx.x / heads, tiles = (vdim + VT - 1) / VT;
    const int b = row0 + part / tiles, c0 = part % tiles * VT, tid = threadIdx.x, p = tid % P, g4 = tid / P * NC;
    const int t0 = query_start[b], n = query_start[b + 1] - t0, blocks = blocks_of(query_start, b, least);
    if (blocks == 0) return;
    int first = 0;                                                       // the row's first block
    for (int a = row0; a < b; ++a) first += blocks_of(query_start, a, least);
    const float* src = scratch + ((size_t)first * heads + h) * FLOATS;
    float* S_g = state + ((size_t)row_slot[b] * heads + h) * vdim * DIM;
    uint64_t S[NC][2 * QUADS];
#pragma unroll
    for (int c = 0; c < NC; ++c)
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const int x = min(c0 + g4 + c, vdim - 1);                    // (columns past the last repeat it and are not written)
            const ulonglong2 w = *(const ulonglong2*)(S_g + (size_t)x * DIM + (i * P + p) * 4);
            S[c][2 * i] = w.x; S[c][2 * i + 1] = w.y;
        }
    auto fetch = [&](int block) {
        float* dst = sm + (block % RB_STAGES) * STAGE;
        const float* from = src + (size_t)block * heads * FLOATS;
        for (int e = tid; e < FLOATS / 4; e += THREADS)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + e * 4)), "l"(from + e * 4) : "memory");
        for (int e = tid; e < T * VT; e += THREADS) {
            const int j = e / VT, x = c0 + e % VT, t = block * T + j;
            const bool there = t < n && x < vdim;
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst + FLOATS + e)),
                         "l"(v + (there ? ((size_t)(t0 + t) * heads + h) * vdim + x : 0)), "r"(there ? 4 : 0) : "memory");
        }
    };
    auto write = [&](int block) {                                        // a block's outputs, a token's columns side by side
        for (int e = tid; e < T * VT; e += THREADS) {
            const int j = e / VT, x = c0 + e % VT, t = block * T + j;
            if (t < n && x < vdim) out[((size_t)(t0 + t) * heads + h) * vdim + x] = so[(block & 1) * T * VT + e];
        }
    };
#pragma unroll
    for (int s = 0; s < RB_STAGES - 1; ++s) {
        if (s < blocks) fetch(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int block = 0; block < blocks; ++block) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(RB_STAGES - 2) : "memory");
        __syncthreads();                                                 // the block is here, the one before has been read
        if (block + RB_STAGES - 1 < blocks) fetch(block + RB_STAGES - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        if (block > 0) write(block - 1);
        const float* kd = sm + (block % RB_STAGES) * STAGE;
        const float* qd = kd + T * DIM;
        const float* kr = qd + T * DIM;
        const float* rr = kr + T * DIM;
        const float* gT = kr + (MODE == RB_GENERAL ? 2 : 1) * T * DIM;
        const float* coef = gT + 2 * DIM;
        float x[NC][V];                                                  // per column: S^T k of the tokens, then S^T q
#pragma unroll
        for (int j = 0; j < T; ++j) {
            uint64_t a[NC], o[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) a[c] = o[c] = 0;
#pragma unroll
            for (int i = 0; i < QUADS; ++i) {
                const int d = j * DIM + (i * P + p) * 4;
                const ulonglong2 q = *(const ulonglong2*)(qd + d), k = *(const ulonglong2*)(kd + d);
#pragma unroll
                for (int c = 0; c < NC; ++c) {
                    rb_fma2(o[c], S[c][2 * i], q.x); rb_fma2(o[c], S[c][2 * i + 1], q.y);
                    rb_fma2(a[c], S[c][2 * i], k.x); rb_fma2(a[c], S[c][2 * i + 1], k.y);
                }
            }
#pragma unroll
            for (int c = 0; c < NC; ++c) { x[c][j] = rb_sum(a[c]); x[c][T + j] = rb_sum(o[c]); }
        }
        const int jo = p & (T - 1);                                      // the token whose read-out this lane completes
        float mine[NC], o[NC], row[T], row2[MODE == RB_GENERAL ? T : 1];
#pragma unroll
        for (int c = 0; c < NC; ++c) o[c] = mine[c] = lanes_sum<V, P>(x[c], p);
#pragma unroll
        for (int i = 0; i < T; i += 4) {
            *(float4*)&row[i] = *(const float4*)(coef + jo * T + i);
            if constexpr (MODE == RB_GENERAL) *(float4*)&row2[i] = *(const float4*)(coef + T * T + jo * T + i);
        }
        uint64_t w[NC][2 * QUADS];                                       // what the block adds to S
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const ulonglong2 g = *(const ulonglong2*)(gT + DIM + (i * P + p) * 4);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                w[c][2 * i] = w[c][2 * i + 1] = 0;
                rb_fma2(w[c][2 * i], S[c][2 * i], g.x);
                rb_fma2(w[c][2 * i + 1], S[c][2 * i + 1], g.y);
            }
        }
#pragma unroll
        for (int j = 0; j < T; ++j) {
            uint64_t u[NC], y[NC];
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float a = __shfl_sync(0xffffffffu, mine[c], j, P), value = kd[FLOATS + j * VT + g4 + c];
                const float d = MODE == RB_DELTA ? value - a : value;
                if (j <= jo) o[c] = fmaf(row[j], d, o[c]);               // (and not zero times a later token's value)
                u[c] = rb_twice(d);
                if constexpr (MODE == RB_GENERAL) { if (j <= jo) o[c] = fmaf(-row2[j], a, o[c]); y[c] = rb_twice(-a); }
            }
#pragma unroll
            for (int i = 0; i < QUADS; ++i) {
                const int d = j * DIM + (i * P + p) * 4;
                const ulonglong2 k = *(const ulonglong2*)(kr + d);
#pragma unroll
                for (int c = 0; c < NC; ++c) { rb_fma2(w[c][2 * i], k.x, u[c]); rb_fma2(w[c][2 * i + 1], k.y, u[c]); }
                if (MODE == RB_GENERAL) {
                    const ulonglong2 r = *(const ulonglong2*)(rr + d);
#pragma unroll
                    for (int c = 0; c < NC; ++c) { rb_fma2(w[c][2 * i], r.x, y[c]); rb_fma2(w[c][2 * i + 1], r.y, y[c]); }
                }
            }
        }
        if (p >= T && p < V) {
#pragma unroll
            for (int c = 0; c < NC; ++c) so[(block & 1) * T * VT + jo * VT + g4 + c] = o[c];
        }
#pragma unroll
        for (int i = 0; i < QUADS; ++i) {
            const ulonglong2 g = *(const ulonglong2*)(gT + (i * P + p) * 4);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                rb_fma2(w[c][2 * i], S[c][2 * i], g.x);
                rb_fma2(w[c][2 * i + 1], S[c][2 * i + 1], g.y);
                S[c][2 * i] = w[c][2 * i]; S[c][2 * i + 1] = w[c][2 * i + 1];
            }
        }
    }
    __syncthreads();
    write(blocks - 1);
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (c0 + g4 + c < vdim)
#pragma unroll
            for (int i = 0; i < QUADS; ++i) {
                ulonglong2 w;
                w.x = S[c][2 * i]; w.y = S[c][2 * i + 1];
                *(ulonglong2*)(S_g + (size_t)(c0 + g4 + c) * DIM + (i * P + p) * 4) = w;
            }
}

// Floats of scratch per block of eight tokens and head; 0: a key size that these kernels do not take.
extern "C" int hb_recurrent_blocks_floats(int general, int dim) {
    if (dim != 64 && dim != 128 && dim != 256) return 0;
    return rb_floats(general ? RB_GENERAL : RB_DELTA, dim);
}

template <int DPT, int P, int NC, int MODE>
static int launch_blocks(float* out, const float* qk, const float* v, const float* decay, const float* head_decay, const float* beta,
                         const float* rate, float* state, float* scratch, const int32_t* query_start, const int32_t* row_slot, int row0,
                         int rows, int blocks, int least, int heads, int kv_heads, int vdim, cudaStream_t s) {
    constexpr int DIM = DPT * P, VT = RB_VT;
    recurrent_block_kernel<DIM / 32, MODE><<<dim3(blocks, (heads + 3) / 4), 128, 0, s>>>(
        scratch, qk, decay, head_decay, beta, rate, query_start, row0, rows, least, heads, kv_heads);
    HB_LAUNCH_CHECK("recurrent_block");
    const int smem = (RB_STAGES * (rb_floats(MODE, DIM) + RB_T * VT) + 2 * RB_T * VT) * (int)sizeof(float);
    auto kernel = recurrent_blocks_kernel<DPT, P, NC, MODE>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<dim3((unsigned)((rows - row0) * ((vdim + VT - 1) / VT) * heads)), P * VT / NC, smem, s>>>(out, scratch, v, state, query_start, row_slot, row0, least, heads, vdim);
    HB_LAUNCH_CHECK("recurrent_blocks");
    return 0;
}

// Those of rows row0 .. rows - 1 of the batch that bring `least` tokens or more, otherwise as hb_recurrent_scan with beta or with rate.
// `taken`: how many these are (or may be), for the choice below; blocks: at least the sum over them of ceil(tokens / 8); scratch: blocks * heads * hb_recurrent_blocks_floats(...) floats on a 16-byte boundary.
extern "C" int hb_recurrent_blocks(float* out, const float* qk, const float* v, const float* decay, const float* head_decay,
                                   const float* beta, const float* rate, float* state, float* scratch, const int32_t* query_start,
                                   const int32_t* row_slot, int row0, int rows, int blocks, int least, int taken,
                                   int heads, int kv_heads, int dim, int vdim, hb_stream stream) {
    if (rows <= row0 || blocks <= 0) return 0;
    if (kv_heads < 1 || heads % kv_heads) HB_REFUSE("recurrent_blocks: %d heads are no multiple of %d key heads", heads, kv_heads);
    if (vdim < 1 || !hb_recurrent_blocks_floats(0, dim)) HB_REFUSE("recurrent_blocks: key size %d (64, 128 or 256), value size %d", dim, vdim);
    if ((decay != nullptr) == (head_decay != nullptr)) HB_REFUSE("recurrent_blocks: give decays per channel and token, or one per head");
    if ((rate != nullptr) == (beta != nullptr) || (rate && !decay)) HB_REFUSE("recurrent_blocks: either a delta rule's beta or, with decays per channel, removal rates");
    if (heads > 65535 || (long)(rows - row0) * heads * ((vdim + RB_VT - 1) / RB_VT) > 0x7fffffffL)
        HB_REFUSE("recurrent_blocks: %d rows, %d heads, value size %d", rows - row0, heads, vdim);
    if ((((uintptr_t)qk | (uintptr_t)decay | (uintptr_t)rate | (uintptr_t)state | (uintptr_t)scratch) & 15) != 0)
        HB_REFUSE("recurrent_blocks: qk, decay, rate, state and scratch must lie on 16-byte boundaries");
    cudaStream_t s = (cudaStream_t)stream;
    // Four columns a thread halve the reads of shared memory a column; two keep an SM's four schedulers busy where there is no more
    // than a CTA or two for each (heads of 128 by 128, the delta rule: 16 heads and 2,048 tokens 304 us with two, 403 with four; 16 heads and
    // rows of 1,500 and 938 tokens 295 and 311; 32 heads and 2,048 tokens 454 and 431; 32 heads and the two rows 529 and 475).
    const bool many = (long)taken * heads * ((vdim + RB_VT - 1) / RB_VT) > 296;
#define RB_ARGS out, qk, v, decay, head_decay, beta, rate, state, scratch, query_start, row_slot, row0, rows, blocks, least, heads, kv_heads, vdim, s
#define RB_GO(D, P) do { \
        if (many) return rate ? launch_blocks<D, P, 4, RB_GENERAL>(RB_ARGS) : launch_blocks<D, P, 4, RB_DELTA>(RB_ARGS); \
        return rate ? launch_blocks<D, P, 2, RB_GENERAL>(RB_ARGS) : launch_blocks<D, P, 2, RB_DELTA>(RB_ARGS); \
    } while (0)
    if (dim == 64) RB_GO(4, 16);
    if (dim == 128) RB_GO(8, 16);
    RB_GO(8, 32);
#undef RB_GO
#undef RB_ARGS
}
