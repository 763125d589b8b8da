// The state-space recurrence, and those of recurrent.cu whose decay is one number per head or per head and token and that have no
// delta rule, for rows of several tokens, in chunks of 64 (the form of Dao and Gu, Transformers are SSMs: Generalized
// Models and Efficient Algorithms Through Structured State Space Duality), everything in 32-bit on CUDA cores:
//     S_t = g_t S_(t-1) + dt_t B_t x_t^T,  y_t = S_t^T C_t + skip x_t,  g_t = exp(-exp(rate_log) dt_t)
// With L_i the sum of the logarithms of g over a chunk's tokens up to i (kept as a pair of float32 whose sum is exact to double
// precision: what the weights need are differences of such sums), a chunk with the state S_in before it gives
//     y_i = sum_(j <= i) (C_i . B_j) exp(L_i - L_j) dt_j x_j + exp(L_i) S_in^T C_i + skip x_i
//     S_out = exp(L_last) S_in + sum_j exp(L_last - L_j) dt_j B_j x_j^T.
// With a decay given as itself (FIXED: one per head, TOKEN: per head and token) dt = 1, there is no skip, and L sums the logarithms of
// its magnitude in double precision, a zero counting as -10^4 (below which an exponential is zero); signs are kept beside it. A value that is no finite
// number reaches the outputs from its token on and no earlier one.
// 2,048 tokens of 16 heads of 128 by 128 with a decay per head: 144 us in chunks, 417 us token by token (recurrent.cu).
// Four kernels: the chunks' products C_i . B_j, per group; the chunks' own contributions to the state, per head; the walk over a
// row's chunks, an element of the state a thread, which leaves every chunk's S_in behind and writes the row's state back; the
// chunks' outputs, per head. Only the third is sequential, one multiply-add a chunk. Blocks find their (row, chunk) in the step's
// rows; launches may have more tiles than the step has chunks. One-token rows: csrc/recurrent.cu.
#include <type_traits>

#include "common.cuh"

#define SS_Q 64                          // tokens a chunk
#define SS_T 64                          // rows and columns of an output tile
#define SS_K 32                          // depth of a staged slice
#define SS_THREADS 128                   // a thread: 8 rows x 4 columns of a tile

struct Chunk { int row, t0, n, first_tile; };              // the batch row, first token, tokens, the row's first tile

// Tiles of row b: ceil(tokens / 64), and none of a row of fewer than `least` tokens.
__device__ __forceinline__ int tiles_of(const int32_t* __restrict__ query_start, int b, int least) {
    const int n = query_start[b + 1] - query_start[b];
    return n >= least ? (n + SS_Q - 1) / SS_Q : 0;
}

// Tile number -> chunk (row -1: there is none). Rows row0 .. rows - 1 in order.
__device__ __forceinline__ Chunk find_chunk(const int32_t* __restrict__ query_start, int row0, int rows, int tile, int least) {
    int left = tile;
    for (int b = row0; b < rows; ++b) {
        const int n = query_start[b + 1] - query_start[b], tiles = tiles_of(query_start, b, least);
        if (left < tiles) return {b, query_start[b] + left * SS_Q, min(SS_Q, n - left * SS_Q), tile - left};
        left -= tiles;
    }
    return {-1, 0, 0, 0};
}

// A slice of an operand in shared memory: element (k, i) in the group of four floats at(k, i / 4). The groups of a row of k are
// permuted by k / 4, so that stores of four k's of one i by eight neighbouring lanes, and of four i's by four, hit different banks.
__device__ __forceinline__ int group_at(int k, int g) { return k * (SS_T / 4) + (g ^ ((k >> 2) & 7)); }

enum Form { STATE_SPACE, FIXED, TOKEN };                   // where decays come from: dt and rate_log; head_decay in rate_log's place; token_decay in dt's

// total += a^T b over a slice. FIXED and TOKEN: 16 steps of k to a sum of their own, since one sum over all steps loses twice as much
// (an output's error against 64 bits 2.5e-7 in place of 1.3e-7, the token-by-token scan's 1.0 to 2.1e-7 for decays of 0.875 to 0.984).
// That takes a second set of sums and so three CTAs an SM in place of four; the state space, whose only form for prompts this is, keeps
// one sum and four (2,048 tokens, 32 heads of 64 over a state of 128: 108 us, 129 us with the sums in parts).
#define SS_CTAS(FORM) ((FORM) == STATE_SPACE ? 4 : 3)
template <int FORM>
__device__ __forceinline__ void tile_step(float (&total)[8][4], const float* a, const float* b, int depth) {
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const float4* a4 = (const float4*)a;
    const float4* b4 = (const float4*)b;
    auto steps = [&](float (&acc)[8][4], int from, int to) {
#pragma unroll 8
        for (int k = from; k < to; ++k) {
            const float4 r0 = a4[group_at(k, ty * 2)], r1 = a4[group_at(k, ty * 2 + 1)], c = b4[group_at(k, tx)];
            const float r[8] = {r0.x, r0.y, r0.z, r0.w, r1.x, r1.y, r1.z, r1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                acc[i][0] = fmaf(r[i], c.x, acc[i][0]); acc[i][1] = fmaf(r[i], c.y, acc[i][1]);
                acc[i][2] = fmaf(r[i], c.z, acc[i][2]); acc[i][3] = fmaf(r[i], c.w, acc[i][3]);
            }
        }
    };
    if constexpr (FORM == STATE_SPACE) steps(total, 0, depth);
    else
        for (int k0 = 0; k0 < depth; k0 += 16) {
            float acc[8][4] = {};
            steps(acc, k0, min(depth, k0 + 16));
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) total[i][j] += acc[i][j];
        }
}

// Slices travel through registers (the next one is on its way while the current one is multiplied), 16 bytes a load: four quads a
// thread and operand. `along`: the operand's memory runs along k (element (row i, k) at p[i * stride + k]); eight neighbouring lanes
// load 128 bytes of one row. `across`: it runs along the tile's rows (element (k, i) at p[k * stride + i]).
struct Quads { float4 v[4]; };
// Which of x (1) and C, B (2) can be read 16 bytes at a time: rows of whole quads that begin on a 16-byte boundary.
static int in_quads(const float* x, int vdim, const float* cb, int n) {
    return (vdim % 4 == 0 && (uintptr_t)x % 16 == 0 ? 1 : 0) | (n % 4 == 0 && (uintptr_t)cb % 16 == 0 ? 2 : 0);
}
__device__ __forceinline__ float4 load_quad(const float* p, int left, bool vec) {        // zeros from `left` on
    if (vec && left >= 4) return *(const float4*)p;
    return make_float4(left > 0 ? p[0] : 0.f, left > 1 ? p[1] : 0.f, left > 2 ? p[2] : 0.f, left > 3 ? p[3] : 0.f);
}
__device__ __forceinline__ void fetch_along(Quads& q, const float* p, size_t stride, int rows, int depth, bool vec) {
    const int i = threadIdx.x >> 3, k = (threadIdx.x & 7) * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) q.v[r] = load_quad(p + (i + 16 * r) * stride + k, i + 16 * r < rows ? depth - k : 0, vec);
}
__device__ __forceinline__ void store_along(float* a, const Quads& q) {
    const int k = (threadIdx.x & 7) * 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const int i = (threadIdx.x >> 3) + 16 * r, g = i >> 2, e = i & 3;      // (k .. k + 3 share their permutation)
        a[group_at(k, g) * 4 + e] = q.v[r].x; a[group_at(k + 1, g) * 4 + e] = q.v[r].y;
        a[group_at(k + 2, g) * 4 + e] = q.v[r].z; a[group_at(k + 3, g) * 4 + e] = q.v[r].w;
    }
}
__device__ __forceinline__ void fetch_across(Quads& q, const float* p, size_t stride, int rows, int depth, bool vec) {
    const int i = (threadIdx.x & 15) * 4, k = threadIdx.x >> 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) q.v[r] = load_quad(p + (k + 8 * r) * stride + i, k + 8 * r < depth ? rows - i : 0, vec);
}
__device__ __forceinline__ void store_across(float* a, const Quads& q) {
    const int k = threadIdx.x >> 4;
#pragma unroll
    for (int r = 0; r < 4; ++r) ((float4*)a)[group_at(k + 8 * r, threadIdx.x & 15)] = q.v[r];
}
__device__ __forceinline__ void scale_quad(float4& v, float f) { v.x *= f; v.y *= f; v.z *= f; v.w *= f; }

// L_i of a chunk's tokens for one head, by warp 0: hi + lo in two floats; tokens past the chunk repeat the last. sign: of the decays'
// product up to i (not for STATE_SPACE).
template <int FORM>
__device__ __forceinline__ void log_decays(float* hi, float* lo, float* steps, float* sign, const float* __restrict__ dt, const Chunk& c,
                                           int heads, int h, const float* __restrict__ rate_log) {
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        const bool in0 = 2 * lane < c.n, in1 = 2 * lane + 1 < c.n;
        float d0 = in0 ? 1.f : 0.f, d1 = in1 ? 1.f : 0.f;
        if (FORM != FIXED) {
            d0 = in0 ? dt[(size_t)(c.t0 + 2 * lane) * heads + h] : 0.f;
            d1 = in1 ? dt[(size_t)(c.t0 + 2 * lane + 1) * heads + h] : 0.f;
        }
        double a0, a1;
        if (FORM == STATE_SPACE) {
            const float rate = expf(rate_log[h]);
            a0 = -(double)rate * d0; a1 = -(double)rate * d1;
        } else {
            const float g0 = FORM == FIXED ? rate_log[h] : d0, g1 = FORM == FIXED ? rate_log[h] : d1;
            auto logarithm = [](float g) -> double {
                const double a = g == 0.f ? -1e4 : log(fabs((double)g));
                return a > 1e4 ? 1e4 : a;
            };
            a0 = in0 ? logarithm(g0) : 0.0; a1 = in1 ? logarithm(g1) : 0.0;
            const unsigned n0 = __ballot_sync(0xffffffffu, in0 && g0 < 0.f), n1 = __ballot_sync(0xffffffffu, in1 && g1 < 0.f);
            const unsigned before = (1u << lane) - 1, here = __popc(n0 & before) + __popc(n1 & before) + ((n0 >> lane) & 1);
            sign[2 * lane] = here & 1 ? -1.f : 1.f;
            sign[2 * lane + 1] = (here + ((n1 >> lane) & 1)) & 1 ? -1.f : 1.f;
            d0 = in0 ? 1.f : 0.f; d1 = in1 ? 1.f : 0.f;
        }
        double s = a0 + a1;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double up = __shfl_up_sync(0xffffffffu, s, o);
            if (lane >= o) s += up;
        }
        const double l0 = s - a1;
        steps[2 * lane] = d0; steps[2 * lane + 1] = d1;
        hi[2 * lane] = (float)l0; lo[2 * lane] = (float)(l0 - (double)(float)l0);
        hi[2 * lane + 1] = (float)s; lo[2 * lane + 1] = (float)(s - (double)(float)s);
    }
}

// ---- products[tile][group][i][j] = C_i . B_j, [64][64] each. grid (tiles, groups)
template <int FORM>
__global__ void __launch_bounds__(SS_THREADS, SS_CTAS(FORM)) ss_products_kernel(float* __restrict__ products, const float* __restrict__ cb,
                                                                 const int32_t* __restrict__ query_start, int row0, int rows, int groups, int n, int quads, int least) {
    __shared__ __align__(16) float a[SS_K * SS_T], b[SS_K * SS_T];
    const Chunk c = find_chunk(query_start, row0, rows, blockIdx.x, least);
    if (c.row < 0) return;
    const int g = blockIdx.y;
    float acc[8][4] = {};
    Quads qa, qb;
    const float* src = cb + ((size_t)c.t0 * 2 * groups + g) * n;
    const size_t stride = (size_t)2 * groups * n;
    const bool vec = quads & 2;
    fetch_along(qa, src, stride, c.n, n, vec);
    fetch_along(qb, src + (size_t)groups * n, stride, c.n, n, vec);
    for (int k0 = 0; k0 < n; k0 += SS_K) {
        store_along(a, qa);
        store_along(b, qb);
        __syncthreads();
        if (k0 + SS_K < n) {
            fetch_along(qa, src + k0 + SS_K, stride, c.n, n - k0 - SS_K, vec);
            fetch_along(qb, src + (size_t)groups * n + k0 + SS_K, stride, c.n, n - k0 - SS_K, vec);
        }
        tile_step<FORM>(acc, a, b, min(SS_K, n - k0));
        __syncthreads();
    }
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    float* out = products + ((size_t)blockIdx.x * groups + g) * SS_Q * SS_Q;
#pragma unroll
    for (int i = 0; i < 8; ++i) *(float4*)(out + (ty * 8 + i) * SS_Q + tx * 4) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
}

// ---- own[tile][head][p][n] = sum_j exp(L_last - L_j) dt_j x_j[p] B_j[n]; last[tile][head] = exp(L_last). grid (tiles, heads, tiles of
// p times tiles of n)
template <int FORM>
__global__ void __launch_bounds__(SS_THREADS, SS_CTAS(FORM)) ss_own_kernel(float* __restrict__ own, float* __restrict__ last, const float* __restrict__ cb,
                                                            const float* __restrict__ x, const float* __restrict__ dt,
                                                            const float* __restrict__ rate_log, const int32_t* __restrict__ query_start,
                                                            int row0, int rows, int heads, int groups, int n, int vdim, int n_tiles, int quads, int least) {
    __shared__ __align__(16) float a[SS_K * SS_T], b[SS_K * SS_T];
    __shared__ float hi[SS_Q], lo[SS_Q], steps[SS_Q], w[SS_Q], sign[FORM == STATE_SPACE ? 1 : SS_Q];
    const Chunk c = find_chunk(query_start, row0, rows, blockIdx.x, least);
    if (c.row < 0) return;
    const int h = blockIdx.y, g = h / (heads / groups);
    const int p0 = ((int)blockIdx.z / n_tiles) * SS_T, n0 = ((int)blockIdx.z % n_tiles) * SS_T;
    Quads qa, qb;
    const size_t xs = (size_t)heads * vdim, bs = (size_t)2 * groups * n;
    const float* xp = x + ((size_t)c.t0 * heads + h) * vdim + p0;
    const float* bp = cb + (((size_t)c.t0 * 2 + 1) * groups + g) * n + n0;
    const bool vx = quads & 1, vb = quads & 2;
    fetch_across(qa, xp, xs, vdim - p0, c.n, vx);                   // (on its way while the decays are added up)
    fetch_across(qb, bp, bs, n - n0, c.n, vb);
    log_decays<FORM>(hi, lo, steps, sign, dt, c, heads, h, rate_log);
    __syncthreads();
    if (threadIdx.x < SS_Q) {
        const int j = threadIdx.x;
        float f = 1.f, all = 1.f;
        if (FORM != STATE_SPACE) { all = sign[SS_Q - 1]; f = all * sign[j]; }
        w[j] = f * expf((hi[SS_Q - 1] - hi[j]) + (lo[SS_Q - 1] - lo[j])) * steps[j];
        if (j == 0 && blockIdx.z == 0) last[(size_t)blockIdx.x * heads + h] = all * expf(hi[SS_Q - 1] + lo[SS_Q - 1]);
    }
    __syncthreads();
    float acc[8][4] = {};
    for (int k0 = 0; k0 < c.n; k0 += SS_K) {
#pragma unroll
        for (int r = 0; r < 4; ++r) scale_quad(qa.v[r], w[min(k0 + ((int)threadIdx.x >> 4) + 8 * r, SS_Q - 1)]);
        store_across(a, qa);
        store_across(b, qb);
        __syncthreads();
        if (k0 + SS_K < c.n) {
            fetch_across(qa, xp + (k0 + SS_K) * xs, xs, vdim - p0, c.n - k0 - SS_K, vx);
            fetch_across(qb, bp + (k0 + SS_K) * bs, bs, n - n0, c.n - k0 - SS_K, vb);
        }
        tile_step<FORM>(acc, a, b, min(SS_K, c.n - k0));
        __syncthreads();
    }
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    float* out = own + ((size_t)blockIdx.x * heads + h) * vdim * n;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int p = p0 + ty * 8 + i, col = n0 + tx * 4;
        if (p >= vdim) break;
        if ((n & 3) == 0 && col + 3 < n) *(float4*)(out + (size_t)p * n + col) = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        else
#pragma unroll
            for (int k = 0; k < 4; ++k) if (col + k < n) out[(size_t)p * n + col + k] = acc[i][k];
    }
}

// ---- a row's chunks in order: own[tile] <- the state before the chunk, state <- the state behind the last. grid (rows - row0, heads,
// slices of the state), an element (V: four) a thread.
template <bool V>
__global__ void ss_walk_kernel(float* __restrict__ own, const float* __restrict__ last, float* __restrict__ state,
                               const int32_t* __restrict__ query_start, const int32_t* __restrict__ row_slot, int row0, int heads, int size,
                               int least) {
    typedef typename std::conditional<V, float4, float>::type E;
    const int b = row0 + (int)blockIdx.x, h = blockIdx.y, e = blockIdx.z * blockDim.x + threadIdx.x;
    int first = 0;
    for (int r = row0; r < b; ++r) first += tiles_of(query_start, r, least);
    const int tiles = tiles_of(query_start, b, least);
    if (e >= (V ? size >> 2 : size) || tiles == 0) return;
    E* st = (E*)(state + ((size_t)row_slot[b] * heads + h) * size) + e;
    const size_t stride = (size_t)heads * size / (V ? 4 : 1);
    E* p = (E*)(own + ((size_t)first * heads + h) * size) + e;
    const float* f = last + (size_t)first * heads + h;
    E s = *st;
    auto step = [&](float d, const E& v) {
        if constexpr (V) { s.x = fmaf(d, s.x, v.x); s.y = fmaf(d, s.y, v.y); s.z = fmaf(d, s.z, v.z); s.w = fmaf(d, s.w, v.w); }
        else s = fmaf(d, s, v);
    };
    int i = 0;
    for (; i + 8 <= tiles; i += 8, p += 8 * stride, f += 8 * (size_t)heads) {        // (eight chunks' loads fly together)
        E v[8];
        float d[8];
#pragma unroll
        for (int k = 0; k < 8; ++k) { v[k] = p[k * stride]; d[k] = f[k * (size_t)heads]; }
#pragma unroll
        for (int k = 0; k < 8; ++k) { p[k * stride] = s; step(d[k], v[k]); }
    }
    for (; i < tiles; ++i, p += stride, f += heads) {
        const E v = p[0];
        p[0] = s;
        step(f[0], v);
    }
    *st = s;
}

// ---- y_i[p] of a chunk: the products' part over its own tokens, the state's part over n, the skip. grid (tiles, heads, tiles of p)
template <int FORM>
__global__ void __launch_bounds__(SS_THREADS, SS_CTAS(FORM)) ss_out_kernel(float* __restrict__ y, const float* __restrict__ products,
                                                            const float* __restrict__ before, const float* __restrict__ cb,
                                                            const float* __restrict__ x, const float* __restrict__ dt,
                                                            const float* __restrict__ rate_log, const float* __restrict__ skip,
                                                            const int32_t* __restrict__ query_start, int row0, int rows, int heads,
                                                            int groups, int n, int vdim, int quads, int least) {
    __shared__ __align__(16) float a[SS_K * SS_T], b[SS_K * SS_T];
    __shared__ float hi[SS_Q], lo[SS_Q], steps[SS_Q], w[SS_Q], sign[FORM == STATE_SPACE ? 1 : SS_Q];
    __shared__ int bad[SS_T];                                       // per column: the first token whose value is no finite number
    const Chunk c = find_chunk(query_start, row0, rows, blockIdx.x, least);
    if (c.row < 0) return;
    const int h = blockIdx.y, g = h / (heads / groups), p0 = (int)blockIdx.z * SS_T;
    const float* cbp = products + ((size_t)blockIdx.x * groups + g) * SS_Q * SS_Q;
    const float* xp = x + ((size_t)c.t0 * heads + h) * vdim + p0;
    const float* cp = cb + ((size_t)c.t0 * 2 * groups + g) * n;
    const float* sp = before + (((size_t)blockIdx.x * heads + h) * vdim + p0) * n;
    const size_t xs = (size_t)heads * vdim, cs = (size_t)2 * groups * n;
    const bool vx = quads & 1, vn = quads & 2;                      // (the state's rows are read as C's are)
    const int own_slices = (c.n + SS_K - 1) / SS_K, slices = own_slices + (n + SS_K - 1) / SS_K;
    Quads qa, qb;
    auto fetch = [&](int s) {
        if (s < own_slices) {                                       // over the chunk's tokens j
            const int k0 = s * SS_K;
            fetch_along(qa, cbp + k0, SS_Q, SS_Q, SS_K, true);
            fetch_across(qb, xp + k0 * xs, xs, vdim - p0, c.n - k0, vx);
        } else {                                                    // over the state's channels
            const int k0 = (s - own_slices) * SS_K;
            fetch_along(qa, cp + k0, cs, c.n, n - k0, vn);
            fetch_along(qb, sp + k0, n, vdim - p0, n - k0, vn);
        }
    };
    fetch(0);                                                       // (on its way while the decays are added up)
    log_decays<FORM>(hi, lo, steps, sign, dt, c, heads, h, rate_log);
    __syncthreads();
    if (threadIdx.x < SS_Q) {
        const int i = threadIdx.x;
        w[i] = (FORM == STATE_SPACE ? 1.f : sign[i]) * expf(hi[i] + lo[i]);
        bad[i] = SS_Q;
    }
    __syncthreads();
    float acc[8][4] = {};
    for (int s = 0; s < slices; ++s) {
        if (s < own_slices) {                                       // weight of token j in row i: C_i . B_j exp(L_i - L_j) dt_j, j <= i
            const int j = s * SS_K + ((int)threadIdx.x & 7) * 4;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const int row = ((int)threadIdx.x >> 3) + 16 * r;
                const float hr = hi[row], lr = lo[row];
                auto weight = [&](int jj, float v) -> float {
                    if (jj > row || jj >= c.n) return 0.f;
                    const float f = FORM == STATE_SPACE ? v : v * (sign[row] * sign[jj]);
                    return f * expf((hr - hi[jj]) + (lr - lo[jj])) * steps[jj];
                };
                qa.v[r].x = weight(j, qa.v[r].x); qa.v[r].y = weight(j + 1, qa.v[r].y);
                qa.v[r].z = weight(j + 2, qa.v[r].z); qa.v[r].w = weight(j + 3, qa.v[r].w);
                float* x4 = &qb.v[r].x;                             // (a weight of zero would make a NaN of an infinity in an earlier row)
                if (!(fabsf(x4[0]) + fabsf(x4[1]) + fabsf(x4[2]) + fabsf(x4[3]) < INFINITY)) {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (!isfinite(x4[e])) {
                            atomicMin(&bad[((int)threadIdx.x & 15) * 4 + e], s * SS_K + ((int)threadIdx.x >> 4) + 8 * r);
                            x4[e] = 0.f;
                        }
                }
            }
        } else {
#pragma unroll
            for (int r = 0; r < 4; ++r) scale_quad(qa.v[r], w[((int)threadIdx.x >> 3) + 16 * r]);
        }
        store_along(a, qa);
        if (s < own_slices) store_across(b, qb); else store_along(b, qb);
        __syncthreads();
        if (s + 1 < slices) fetch(s + 1);
        // (the second half of a chunk's tokens weighs nothing in its first half's rows)
        if (s >= own_slices || s == 0 || (int)(threadIdx.x >> 5) * 16 + 15 >= s * SS_K) tile_step<FORM>(acc, a, b, SS_K);
        __syncthreads();
    }
    const int ty = threadIdx.x >> 4, tx = threadIdx.x & 15;
    const float d = skip ? skip[h] : 0.f;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int r = ty * 8 + i;
        if (r >= c.n) break;
        const size_t at = ((size_t)(c.t0 + r) * heads + h) * vdim + p0 + tx * 4;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if (p0 + tx * 4 + k < vdim) {
                const float v = r >= bad[tx * 4 + k] ? NAN : acc[i][k];
                y[at + k] = skip ? fmaf(d, x[at + k], v) : v;
            }
    }
}

extern "C" size_t hb_state_space_prompt_scratch_floats(int tiles, int heads, int groups, int n, int vdim) {
    return (size_t)tiles * ((size_t)heads * vdim * n + (size_t)groups * SS_Q * SS_Q + heads);
}

template <int FORM>
static int run_chunks(const char* what, float* y, const float* cb, const float* x, const float* dt, const float* rate_log, const float* skip,
                                     float* state, float* scratch, const int32_t* query_start, const int32_t* row_slot, int row0,
                                     int rows, int tiles, int heads, int groups, int n, int vdim, int least, hb_stream stream) {
    if (rows <= row0 || tiles == 0) return 0;
    if (groups < 1 || heads % groups || n < 1 || vdim < 1) HB_REFUSE("%s: %d heads of %d, %d groups of %d", what, heads, vdim, groups, n);
    if (!scratch || ((uintptr_t)scratch & 15) || ((uintptr_t)state & 15)) HB_REFUSE("%s: scratch and state must lie on 16-byte boundaries", what);
    const int p_tiles = (vdim + SS_T - 1) / SS_T, n_tiles = (n + SS_T - 1) / SS_T;
    if (heads > 65535 || (long)p_tiles * n_tiles > 65535) HB_REFUSE("%s: %d heads of %d x %d", what, heads, vdim, n);
    const int size = vdim * n, quads = in_quads(x, vdim, cb, n);
    float* products = scratch;                                     // [tiles][groups][64][64]
    float* own = products + (size_t)tiles * groups * SS_Q * SS_Q;  // [tiles][heads][vdim][n]
    float* last = own + (size_t)tiles * heads * size;              // [tiles][heads]
    cudaStream_t s = (cudaStream_t)stream;
    ss_products_kernel<FORM><<<dim3(tiles, groups), SS_THREADS, 0, s>>>(products, cb, query_start, row0, rows, groups, n, quads, least);
    HB_LAUNCH_CHECK("state_space_products");
    ss_own_kernel<FORM><<<dim3(tiles, heads, p_tiles * n_tiles), SS_THREADS, 0, s>>>(own, last, cb, x, dt, rate_log, query_start, row0, rows, heads,
                                                                               groups, n, vdim, n_tiles, quads, least);
    HB_LAUNCH_CHECK("state_space_own");
    const bool vec = size % 4 == 0;
    const int elements = vec ? size / 4 : size, slices = (elements + 127) / 128;
    if (slices > 65535) HB_REFUSE("%s: states of %d numbers", what, size);
    if (vec) ss_walk_kernel<true><<<dim3(rows - row0, heads, slices), 128, 0, s>>>(own, last, state, query_start, row_slot, row0, heads, size, least);
    else ss_walk_kernel<false><<<dim3(rows - row0, heads, slices), 128, 0, s>>>(own, last, state, query_start, row_slot, row0, heads, size, least);
    HB_LAUNCH_CHECK("state_space_walk");
    ss_out_kernel<FORM><<<dim3(tiles, heads, p_tiles), SS_THREADS, 0, s>>>(y, products, own, cb, x, dt, rate_log, skip, query_start, row0, rows, heads,
                                                                     groups, n, vdim, quads, least);
    HB_LAUNCH_CHECK("state_space_out");
    return 0;
}

extern "C" int hb_state_space_prompt(float* y, const float* cb, const float* x, const float* dt, const float* rate_log, const float* skip,
                                     float* state, float* scratch, const int32_t* query_start, const int32_t* row_slot, int row0,
                                     int rows, int tiles, int heads, int groups, int n, int vdim, hb_stream stream) {
    return run_chunks<STATE_SPACE>("state_space_prompt", y, cb, x, dt, rate_log, skip, state, scratch, query_start, row_slot, row0, rows, tiles,
                                   heads, groups, n, vdim, 1, stream);
}

// hb_recurrent_scan for those of rows row0 .. rows - 1 that bring `least` tokens or more, with one decay per head (head_decay) or per head and token (token_decay) and no delta rule:
// qk [tokens, 2, kv_heads, dim]. tiles and scratch as above, with kv_heads and dim in the places of groups and n.
extern "C" int hb_recurrent_chunks(float* out, const float* qk, const float* v, const float* head_decay, const float* token_decay,
                                   float* state, float* scratch, const int32_t* query_start, const int32_t* row_slot, int row0,
                                   int rows, int tiles, int least, int heads, int kv_heads, int dim, int vdim, hb_stream stream) {
    if ((head_decay != nullptr) == (token_decay != nullptr)) HB_REFUSE("recurrent_chunks: one decay per head, or one per head and token");
    if ((uintptr_t)qk & 15) HB_REFUSE("recurrent_chunks: qk must lie on a 16-byte boundary");
    if (token_decay)
        return run_chunks<TOKEN>("recurrent_chunks", out, qk, v, token_decay, nullptr, nullptr, state, scratch, query_start, row_slot, row0,
                                 rows, tiles, heads, kv_heads, dim, vdim, least, stream);
    return run_chunks<FIXED>("recurrent_chunks", out, qk, v, nullptr, head_decay, nullptr, state, scratch, query_start, row_slot, row0, rows,
                             tiles, heads, kv_heads, dim, vdim, least, stream);
}
