// Paged attention in true 32-bit for head sizes up to 256 that are multiples of 4: the float32 engine's. CUDA cores, no
// reduced precision; what attention_generic.cu computes, with the keys and values of a step read by tiles instead of once
// per query and head, and a lane's reads 16 bytes wide and side by side.
//
// Rows of one token (rows 0 .. n_decode - 1): a cluster of eight blocks per (row, kv head, up to HEADS of its query heads); eight
// lanes share a key and the 256 such groups of lanes of a cluster walk the row's keys, each with a softmax of its own, merged
// per block and then through distributed shared memory.
// Rows of several tokens: a block per (64 queries, head); 64 keys at a time in shared memory, 4 x 4 scores a thread, then
// 4 rows x D / 16 columns of the output. 15 % of the multiply-adds' rate: a tile's keys, then its values, are loaded between barriers with
// nothing in flight beside the arithmetic.
// Measured on 28 layers of 16 heads of 128 over 8 kv heads, two prompts of 333 and 208 tokens and four steps behind them: 95 us
// a layer for the prompts, 9.7 us for the two one-token rows (18.8 with one block in a cluster's place); a warp per query and head, a lane per key, took 755 us on
// average over both.
// Which groups or tiles a key falls into depends on its position alone, so a token's result does not depend on the rows
// beside it nor on where its prompt was cut into portions of two tokens and more (a portion of one goes to the other kernel, whose
// order of the keys is another).
// A key that scores minus infinity (its product with the query overflowed) weighs nothing; a query whose keys all do has no answer: NaN.
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

#define F32_ATT_THREADS 256
#define F32_ATT_PARTS 8

struct F32Rows {
    float* out;
    const float* q;
    const float* kv;
    const int32_t *block_table, *row_slot, *query_start, *kv_len;
    const float* sinks;
    int table_stride, heads, kv_heads, head_dim, pages, page_size, window;
    float scale;
};

__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ void mul2(uint64_t& d, uint64_t a) { asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(d) : "l"(a)); }
__device__ __forceinline__ uint64_t pair(float x, float y) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
    return r;
}
__device__ __forceinline__ float2 halves(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// Offset of the row of key j of a kv head in the pool, or -1 where the table names no page of it.
__device__ __forceinline__ long key_row(const F32Rows& a, const int32_t* table, int j, int hk) {
    const int block = j / a.page_size, page = table[block];
    if (page < 0 || page >= a.pages) return -1;
    return ((((long)page * 2) * a.kv_heads + hk) * a.page_size + (j - block * a.page_size)) * a.head_dim;
}

// ---------------------------------------------------------------- rows of one token
// Bound by the latency of a key's reads: a group fetches its next key's row and value while it works on the one before.
template <int D, int HEADS>                 // D: head_dim rounded up to a multiple of 32 (the lanes' share: D / 8 numbers)
__global__ void __launch_bounds__(F32_ATT_THREADS) attention_f32_decode_kernel(const F32Rows a) {
    constexpr int N = D / 32, GROUPS = F32_ATT_THREADS / 8, ALL = GROUPS * F32_ATT_PARTS;   // N: 16-byte pieces of a row a lane holds
    __shared__ __align__(16) float qs[HEADS][D];
    __shared__ float merge_m[HEADS][GROUPS], merge_l[HEADS][GROUPS];
    __shared__ __align__(16) float sums[GROUPS / 4][D];
    __shared__ float part_m[HEADS], part_l[HEADS], part_v[HEADS][D];
    __shared__ int part_seen;                                            // whether this block met a key at all
    const int per_kv = a.heads / a.kv_heads, chunks = (per_kv + HEADS - 1) / HEADS;
    const int b = blockIdx.y, part = blockIdx.x, hk = blockIdx.z / chunks, h0 = hk * per_kv + blockIdx.z % chunks * HEADS;
    const int count = min(HEADS, (hk + 1) * per_kv - h0);
    const int tid = threadIdx.x, lane = tid & 31, group = tid >> 3, sub = tid & 7;
    const int n = a.kv_len[b], t = a.query_start[b];
    const int pos = n - 1;
    float* o = a.out + ((size_t)t * a.heads + h0) * a.head_dim;
    if (n <= 0) {                                                        // (all blocks of the cluster alike)
        if (part == 0)
            for (int i = tid; i < count * a.head_dim; i += F32_ATT_THREADS) o[i] = 0.f;
        return;
    }
    const float* qr = a.q + ((size_t)t * a.heads + h0) * a.head_dim;
    for (int i = tid; i < HEADS * D; i += F32_ATT_THREADS) {
        const int h = i / D, d = i % D;
        qs[h][d] = h < count && d < a.head_dim ? qr[(size_t)h * a.head_dim + d] * a.scale : 0.f;
    }
    __syncthreads();
    const int32_t* table = a.block_table + (size_t)a.row_slot[b] * a.table_stride;
    const int first = a.window > 0 ? max(0, pos - a.window + 1) : 0;
    const long v_shift = (long)a.kv_heads * a.page_size * a.head_dim;
    float m[HEADS], l[HEADS];
    uint64_t acc[HEADS][2 * N];
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
        m[h] = -INFINITY;
        l[h] = 0.f;
#pragma unroll
        for (int i = 0; i < 2 * N; ++i) acc[h][i] = 0;
    }
    ulonglong2 kn[N], vn[N];
    long base;
    auto fetch = [&](int j) {
        base = j <= pos ? key_row(a, table, j, hk) : -1;
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const int d = (sub + 8 * i) * 4;
            kn[i] = vn[i] = make_ulonglong2(0, 0);
            if (base >= 0 && d < a.head_dim) {
                kn[i] = *(const ulonglong2*)(a.kv + base + d);
                vn[i] = *(const ulonglong2*)(a.kv + base + v_shift + d);
            }
        }
    };
    // the group of a key: its position mod ALL, wherever the window begins
    int j = first - first % ALL + part * GROUPS + group;
    if (j < first) j += ALL;
    const int rounds = (pos - first) / ALL + 1;                         // (the same for all lanes of a warp)
    bool seen = false;
    fetch(j);
    for (int round = 0; round < rounds; ++round) {
        ulonglong2 k[N], v[N];
        const bool there = base >= 0;
        seen |= there;
#pragma unroll
        for (int i = 0; i < N; ++i) { k[i] = kn[i]; v[i] = vn[i]; }
        j += ALL;
        fetch(j);
#pragma unroll
        for (int h = 0; h < HEADS; ++h) {
            uint64_t dot = 0;
#pragma unroll
            for (int i = 0; i < N; ++i) {
                const ulonglong2 qv = *(const ulonglong2*)&qs[h][(sub + 8 * i) * 4];
                fma2(dot, qv.x, k[i].x);
                fma2(dot, qv.y, k[i].y);
            }
            const float2 d2 = halves(dot);
            float s = d2.x + d2.y;
            s += __shfl_xor_sync(0xffffffffu, s, 1);
            s += __shfl_xor_sync(0xffffffffu, s, 2);
            s += __shfl_xor_sync(0xffffffffu, s, 4);
            if (!there) continue;
            const float m_new = fmaxf(m[h], s);
            const float corr = m_new == -INFINITY ? 1.f : expf(m[h] - m_new), p = expf(s - (m_new == -INFINITY ? 0.f : m_new));
            l[h] = l[h] * corr + p;
            m[h] = m_new;
            const uint64_t cc = pair(corr, corr), pp = pair(p, p);
#pragma unroll
            for (int i = 0; i < N; ++i) {
                mul2(acc[h][2 * i], cc);
                mul2(acc[h][2 * i + 1], cc);
                fma2(acc[h][2 * i], pp, v[i].x);
                fma2(acc[h][2 * i + 1], pp, v[i].y);
            }
        }
    }
    if (sub == 0)
#pragma unroll
        for (int h = 0; h < HEADS; ++h) { merge_m[h][group] = m[h]; merge_l[h][group] = l[h]; }
    const int any = __syncthreads_or(seen);
    if (tid == 0) part_seen = any;
#pragma unroll
    for (int h = 0; h < HEADS; ++h) {
        if (h >= count) break;
        const float top = warp_max(merge_m[h][lane]);                    // GROUPS == 32: a lane per group
        const float mine = merge_m[h][lane] == -INFINITY ? 0.f : expf(merge_m[h][lane] - top);
        const float total = warp_sum(merge_l[h][lane] * mine);
        const float f = m[h] == -INFINITY ? 0.f : expf(m[h] - top);
        if (tid == 0) { part_m[h] = top; part_l[h] = total; }
        __syncthreads();                                                 // the head before has been read
#pragma unroll
        for (int i = 0; i < N; ++i) {
            const float2 x = halves(acc[h][2 * i]), y = halves(acc[h][2 * i + 1]);
            float v[4] = {x.x, x.y, y.x, y.y};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                v[c] *= f;                                               // (a group without keys holds zeros)
                v[c] += __shfl_xor_sync(0xffffffffu, v[c], 8);
                v[c] += __shfl_xor_sync(0xffffffffu, v[c], 16);
            }
            if (lane < 8) *(float4*)&sums[tid >> 5][(sub + 8 * i) * 4] = make_float4(v[0], v[1], v[2], v[3]);
        }
        __syncthreads();
        for (int d = tid; d < a.head_dim; d += F32_ATT_THREADS) {
            float s = 0.f;
#pragma unroll
            for (int g = 0; g < GROUPS / 4; ++g) s += sums[g][d];
            part_v[h][d] = s;
        }
    }
    cg::cluster_group cluster = cg::this_cluster();
    cluster.sync();
    for (int i = part * F32_ATT_THREADS + tid; i < count * a.head_dim; i += F32_ATT_PARTS * F32_ATT_THREADS) {
        const int h = i / a.head_dim, d = i - h * a.head_dim;
        float pm[F32_ATT_PARTS], top = -INFINITY, total = 0.f, s = 0.f;
#pragma unroll
        for (int r = 0; r < F32_ATT_PARTS; ++r) { pm[r] = *cluster.map_shared_rank(&part_m[h], r); top = fmaxf(top, pm[r]); }
#pragma unroll
        for (int r = 0; r < F32_ATT_PARTS; ++r) {
            const float f = pm[r] == -INFINITY ? 0.f : expf(pm[r] - top);
            total += *cluster.map_shared_rank(&part_l[h], r) * f;
            s += *cluster.map_shared_rank(&part_v[h][d], r) * f;
        }
        if (a.sinks && total > 0.f) total += expf(a.sinks[h0 + h] - top);
        float inv = 1.f / total;
        if (!(total > 0.f)) {
            int met = 0;
            for (int r = 0; r < F32_ATT_PARTS; ++r) met |= *cluster.map_shared_rank(&part_seen, r);
            inv = met ? NAN : 0.f;
        }
        o[(size_t)h * a.head_dim + d] = s * inv;
    }
    cluster.sync();                                                      // nobody leaves while its sums are being read
}

// ---------------------------------------------------------------- rows of several tokens
#define F32_ATT_TILE 64

template <int D>                            // head_dim rounded up to 64, 128 or 256
__global__ void __launch_bounds__(F32_ATT_THREADS) attention_f32_prompt_kernel(const F32Rows a, int row0, int row1) {
    constexpr int T = F32_ATT_TILE, COLS = D / 64, STRIDE = D + 4;      // a thread's 16-byte columns of the output
    extern __shared__ float4 smem4[];
    float* qs = (float*)smem4;                                           // [T][D]
    float* ks = qs + T * D;                                              // [T][STRIDE]: keys, then values
    float* ps = ks + T * STRIDE;                                         // [T][T + 4]
    __shared__ long bases[T];
    int tile = blockIdx.x, b = row0;
    for (; b < row1; ++b) {                                              // the row this tile belongs to
        const int tiles = (a.query_start[b + 1] - a.query_start[b] + T - 1) / T;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (b >= row1) return;
    const int h = blockIdx.y, hk = h / (a.heads / a.kv_heads), tid = threadIdx.x, ty = tid >> 4, tx = tid & 15;
    const int t0 = a.query_start[b] + tile * T, queries = min(T, a.query_start[b + 1] - t0);
    const int n = a.kv_len[b], pos0 = n - a.query_start[b + 1] + t0;     // the first query's position
    const int32_t* table = a.block_table + (size_t)a.row_slot[b] * a.table_stride;
    const long v_shift = (long)a.kv_heads * a.page_size * a.head_dim;
    for (int i = tid; i < T * (D / 4); i += F32_ATT_THREADS) {
        const int r = i / (D / 4), d = i % (D / 4) * 4;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (r < queries && d < a.head_dim) v = *(const float4*)(a.q + ((size_t)(t0 + r) * a.heads + h) * a.head_dim + d);
        *(float4*)&qs[r * D + d] = make_float4(v.x * a.scale, v.y * a.scale, v.z * a.scale, v.w * a.scale);
    }
    float m[4], l[4];
    uint64_t acc[4][2 * COLS];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = -INFINITY;
        l[i] = 0.f;
#pragma unroll
        for (int c = 0; c < 2 * COLS; ++c) acc[i][c] = 0;
    }
    unsigned met = 0;                                                    // bit i: query i met one of this thread's keys
    const int last = n > 0 ? pos0 + queries - 1 : -1;                    // the last key any of these queries sees
    const int first = a.window > 0 ? max(0, pos0 - a.window + 1) : 0;
    for (int j0 = first - first % T; j0 <= last; j0 += T) {
        __syncthreads();                                                 // the tile before has been read
        if (tid < T) bases[tid] = j0 + tid <= last && j0 + tid >= first ? key_row(a, table, j0 + tid, hk) : -1;
        __syncthreads();
        for (int i = tid; i < T * (D / 4); i += F32_ATT_THREADS) {
            const int r = i / (D / 4), d = i % (D / 4) * 4;
            const long base = bases[r];
            *(float4*)&ks[r * STRIDE + d] = base >= 0 && d < a.head_dim ? *(const float4*)(a.kv + base + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        __syncthreads();
        uint64_t dots[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) dots[i][c] = 0;
#pragma unroll 4
        for (int d = 0; d < D; d += 4) {
            ulonglong2 qv[4], kv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) qv[i] = *(const ulonglong2*)&qs[(ty * 4 + i) * D + d];
#pragma unroll
            for (int c = 0; c < 4; ++c) kv[c] = *(const ulonglong2*)&ks[(tx + 16 * c) * STRIDE + d];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    fma2(dots[i][c], qv[i].x, kv[c].x);
                    fma2(dots[i][c], qv[i].y, kv[c].y);
                }
        }
        __syncthreads();                                                 // the keys have been read: the values take their place
        for (int i = tid; i < T * (D / 4); i += F32_ATT_THREADS) {
            const int r = i / (D / 4), d = i % (D / 4) * 4;
            const long base = bases[r];
            *(float4*)&ks[r * STRIDE + d] = base >= 0 && d < a.head_dim ? *(const float4*)(a.kv + base + v_shift + d) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int pos = pos0 + ty * 4 + i;
            float s[4], top = -INFINITY;
            bool seen[4];
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int j = j0 + tx + 16 * c;
                seen[c] = j <= pos && (a.window <= 0 || pos - j < a.window) && bases[tx + 16 * c] >= 0;
                const float2 d2 = halves(dots[i][c]);
                s[c] = seen[c] ? d2.x + d2.y : -INFINITY;
                if (seen[c]) met |= 1u << i;
                top = fmaxf(top, s[c]);
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float m_new = fmaxf(m[i], top);
            const float corr = m_new == -INFINITY ? 1.f : expf(m[i] - m_new), ref = m_new == -INFINITY ? 0.f : m_new;
            float sum = 0.f;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const float p = expf(s[c] - ref);                        // (0 for what is not seen)
                ps[(ty * 4 + i) * (T + 4) + tx + 16 * c] = p;
                sum += p;
            }
#pragma unroll
            for (int x = 8; x > 0; x >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, x);
            l[i] = l[i] * corr + sum;
            m[i] = m_new;
            const uint64_t cc = pair(corr, corr);
#pragma unroll
            for (int c = 0; c < 2 * COLS; ++c) mul2(acc[i][c], cc);
        }
        __syncthreads();
        // Where some query does not see all keys of the tile, a key it does not see is left out and not multiplied by
        // zero: its value may be an infinity.
        const bool all = j0 + T - 1 <= pos0 && (a.window <= 0 || pos0 + queries - 1 - j0 < a.window);
        if (all) {
#pragma unroll 2
            for (int j = 0; j < T; j += 4) {
                float p[4][4];
#pragma unroll
                for (int i = 0; i < 4; ++i) *(float4*)p[i] = *(const float4*)&ps[(ty * 4 + i) * (T + 4) + j];
#pragma unroll
                for (int jj = 0; jj < 4; ++jj) {
                    ulonglong2 v[COLS];
#pragma unroll
                    for (int c = 0; c < COLS; ++c) v[c] = *(const ulonglong2*)&ks[(j + jj) * STRIDE + tx * 4 + 64 * c];
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        const uint64_t pp = pair(p[i][jj], p[i][jj]);
#pragma unroll
                        for (int c = 0; c < COLS; ++c) {
                            fma2(acc[i][2 * c], pp, v[c].x);
                            fma2(acc[i][2 * c + 1], pp, v[c].y);
                        }
                    }
                }
            }
        } else {
            for (int j = 0; j < T; ++j) {
                ulonglong2 v[COLS];
#pragma unroll
                for (int c = 0; c < COLS; ++c) v[c] = *(const ulonglong2*)&ks[j * STRIDE + tx * 4 + 64 * c];
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const int pos = pos0 + ty * 4 + i;
                    if (j0 + j > pos || (a.window > 0 && pos - j0 - j >= a.window)) continue;
                    const float p = ps[(ty * 4 + i) * (T + 4) + j];
                    const uint64_t pp = pair(p, p);
#pragma unroll
                    for (int c = 0; c < COLS; ++c) {
                        fma2(acc[i][2 * c], pp, v[c].x);
                        fma2(acc[i][2 * c + 1], pp, v[c].y);
                    }
                }
            }
        }
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        const unsigned both = __ballot_sync(0xffffffffu, met >> i & 1);  // of the two queries whose lanes share this warp
        if (r >= queries) continue;
        if (a.sinks && l[i] > 0.f) l[i] += expf(a.sinks[h] - m[i]);
        const float inv = l[i] > 0.f ? 1.f / l[i] : both >> (tid & 16) & 0xffff ? NAN : 0.f;
        float* o = a.out + ((size_t)(t0 + r) * a.heads + h) * a.head_dim;
#pragma unroll
        for (int c = 0; c < COLS; ++c) {
            const int d = tx * 4 + 64 * c;
            if (d >= a.head_dim) continue;
            const float2 x = halves(acc[i][2 * c]), y = halves(acc[i][2 * c + 1]);
            *(float4*)(o + d) = make_float4(x.x * inv, x.y * inv, y.x * inv, y.y * inv);
        }
    }
}

template <int D, int HEADS>
static int launch_decode(const F32Rows& a, int rows, cudaStream_t s) {
    const int per_kv = a.heads / a.kv_heads;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(F32_ATT_PARTS, rows, a.kv_heads * ((per_kv + HEADS - 1) / HEADS));
    config.blockDim = dim3(F32_ATT_THREADS);
    config.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = F32_ATT_PARTS;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = 1;
    HB_CUDA(cudaLaunchKernelEx(&config, attention_f32_decode_kernel<D, HEADS>, a));
    return 0;
}

template <int D>
static int launch_prompt(const F32Rows& a, int row0, int row1, int tiles, cudaStream_t s) {
    const int smem = (F32_ATT_TILE * (2 * D + 4) + F32_ATT_TILE * (F32_ATT_TILE + 4)) * (int)sizeof(float);
    HB_CUDA(cudaFuncSetAttribute(attention_f32_prompt_kernel<D>, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    attention_f32_prompt_kernel<D><<<dim3(tiles, a.heads), F32_ATT_THREADS, smem, s>>>(a, row0, row1);
    return 0;
}

// `tiles`: at least the tiles of 64 queries of the rows from n_decode on. out, q and kv lie on 16-byte boundaries.
extern "C" int hb_attention_f32(float* out, const float* q, const float* kv, const int32_t* block_table, int table_stride,
                                const int32_t* row_slot, const int32_t* query_start, const int32_t* kv_len, int n_decode,
                                int rows, int tiles, int heads, int kv_heads, int head_dim, int pages, int page_size,
                                float scale, int window, const float* sinks, hb_stream stream) {
    if (rows == 0) return 0;
    if (head_dim > 256 || head_dim < 4 || head_dim % 4) HB_REFUSE("attention_f32: head_dim %d is no multiple of 4 up to 256", head_dim);
    if (kv_heads < 1 || heads % kv_heads) HB_REFUSE("attention_f32: %d heads are no multiple of %d kv heads", heads, kv_heads);
    if (((uintptr_t)out | (uintptr_t)q | (uintptr_t)kv) % 16) HB_REFUSE("attention_f32: out, q and kv must lie on 16-byte boundaries");
    if (heads > 65535) HB_REFUSE("attention_f32: %d heads", heads);
    cudaStream_t s = (cudaStream_t)stream;
    F32Rows a = {out, q, kv, block_table, row_slot, query_start, kv_len, sinks,
                 table_stride, heads, kv_heads, head_dim, pages, page_size, window, scale};
    const int per_kv = heads / kv_heads;
    if (n_decode > 65535) HB_REFUSE("attention_f32: %d rows of one token are above 65535", n_decode);
    if (n_decode > 0) {
        const int rc = head_dim <= 64 ? (per_kv == 1 ? launch_decode<64, 1>(a, n_decode, s) : launch_decode<64, 4>(a, n_decode, s))
                     : head_dim <= 128 ? (per_kv == 1 ? launch_decode<128, 1>(a, n_decode, s)
                                          : per_kv == 2 ? launch_decode<128, 2>(a, n_decode, s) : launch_decode<128, 4>(a, n_decode, s))
                     : per_kv == 1 ? launch_decode<256, 1>(a, n_decode, s) : launch_decode<256, 2>(a, n_decode, s);
        if (rc) return rc;
    }
    if (rows > n_decode && tiles > 0) {
        const int rc = head_dim <= 64 ? launch_prompt<64>(a, n_decode, rows, tiles, s)
                     : head_dim <= 128 ? launch_prompt<128>(a, n_decode, rows, tiles, s)
                                       : launch_prompt<256>(a, n_decode, rows, tiles, s);
        if (rc) return rc;
    }
    HB_LAUNCH_CHECK("attention_f32");
    return 0;
}
