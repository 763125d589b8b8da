// Latent attention of prompt portions in bfloat16 on tcgen05 tensor cores, over keys and values that are made per head first.
//
// Folded queries (csrc/latent_tcgen05.cu) spare a decode step the keys and values, but cost a prompt 2 rank + rot multiply-adds a
// query, key and head where a head's own key and value take dim + rot + vdim (1,088 against 320 at rank 512, 128 + 64, 128). So the
// cache rows that a step's portions see are gathered into contiguous rows [latent | rotated part] (hb_latent_gather: every
// request's rows from its window's first on, padded to whole tiles of 64 by zeros), one product with [W_uk; W_uv] makes every
// head's keys and values of them, and this kernel attends: csrc/attention_tcgen05.cu's walk (256 queries of one head a CTA as
// two groups of 128, 64-key tiles by TMA, scores and output in tensor memory, softmax one row per thread, weights back to tensor
// memory, a maximum that lags by up to 2^8) with queries and keys in two parts, the head's own (dim) and the rotated one (rot), which all heads share.
// A tile step's score MMAs are half again as many as without the rotated part, and issuing is what bounds a thread of
// them, so each group has a thread of its own for the scores and one thread does both groups' P V.
// Gather, product and attention of 2,048 tokens, 16 heads of 128 + 64, rank 512: 59 us (the folded form with its two products: 237); of 512
// tokens behind 3,584: 97 (227); 2,048 tokens, 40 heads of 64 + 32, rank 256: 72 (202); 17 tokens: 12 (17).
// Every mbarrier wait is bounded (tcgen05.cuh).
#include "tcgen05.cuh"

#define LX_BM 128                                 // queries a group
#define LX_BN 64                                  // keys a tile
#define LX_STAGES 3
#define LX_BLOCK (64 * 128)                       // bytes of a [64 x 64] block; a [128 x 64] one is two
#define LX_TMEM_COLS 512                          // per group: S0 [0, 64), S1 [64, 128), O [128, 128 + vdim)
#define LX_RESCALE 8.0f
#define LX_THREADS 384

// First key of a request's gathered rows, and how many rows it has there.
__device__ __forceinline__ int lx_first(int n, int nq, int window) { return window > 0 ? max(0, n - nq - window + 1) / LX_BN * LX_BN : 0; }
__device__ __forceinline__ int lx_rows(int n, int nq, int window) { return (n - lx_first(n, nq, window) + LX_BN - 1) / LX_BN * LX_BN; }

// out [total, dk]: the gathered rows of requests row0 .. rows - 1, one after the other. A warp a row, eight rows a block.
__global__ void latent_gather_kernel(bf16* __restrict__ out, const bf16* __restrict__ cache, const int32_t* __restrict__ block_table,
                                     int table_stride, const int32_t* __restrict__ row_slot, const int32_t* __restrict__ query_start,
                                     const int32_t* __restrict__ kv_len, int row0, int rows, int dk, int pages, int page_size,
                                     int window, long total) {
    __shared__ int s_row, s_key;
    const long r0 = (long)blockIdx.x * 8;
    if (threadIdx.x == 0) {
        long left = r0;
        int b = row0;
        for (; b < rows; ++b) {
            const int have = lx_rows(kv_len[b], query_start[b + 1] - query_start[b], window);
            if (left < have) break;
            left -= have;
        }
        s_row = b;
        s_key = b < rows ? (int)left + lx_first(kv_len[b], query_start[b + 1] - query_start[b], window) : 0;
    }
    __syncthreads();
    const int b = s_row, warp = threadIdx.x >> 5, lane = threadIdx.x & 31, key = s_key + warp;
    const long r = r0 + warp;
    if (r >= total) return;
    const uint4* src = nullptr;
    if (b < rows && key < kv_len[b]) {
        const int page = block_table[(size_t)row_slot[b] * table_stride + key / page_size];
        if (page >= 0 && page < pages) src = (const uint4*)(cache + ((size_t)page * page_size + key % page_size) * dk);
    }
    uint4* dst = (uint4*)(out + (size_t)r * dk);
    for (int i = lane; i < dk / 8; i += 32) dst[i] = src ? __ldg(src + i) : make_uint4(0, 0, 0, 0);
}

template <int DIM, int ROT, int VDIM>
__global__ void __launch_bounds__(LX_THREADS, 1) latent_prompt_kernel(
        const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_qr, const __grid_constant__ CUtensorMap map_kv,
        const __grid_constant__ CUtensorMap map_r, bf16* __restrict__ out, const int32_t* __restrict__ query_start,
        const int32_t* __restrict__ kv_len, int row0, int rows, int heads, int q_stride, int qr_stride, int qr_at, int rank,
        float scale_log2, int window, int tile_q, const float* __restrict__ sinks) {
    constexpr int DB = DIM / 64, VB = VDIM / 64, QB = DB + 1;          // blocks of 64 columns: own part, values, both query parts
    constexpr uint32_t Q_BYTES = QB * 2 * LX_BLOCK, STAGE = (DB + 1 + VB) * LX_BLOCK;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const uint32_t q_s = base, kv_s = q_s + 2 * Q_BYTES;
    __shared__ __align__(8) uint64_t bars[1 + 2 * LX_STAGES + 14];
    __shared__ uint32_t s_tmem;
    __shared__ int s_row, s_q0, s_at;
    const uint32_t q_full = smem_addr(bars), kv_full0 = q_full + 8, kv_empty0 = kv_full0 + 8 * LX_STAGES;
    // per group g and buffer i, at index (g * 2 + i): scores computed; weights written; weights read (O holds the tile)
    const uint32_t s_full0 = kv_empty0 + 8 * LX_STAGES, p_full0 = s_full0 + 32, p_empty0 = p_full0 + 32, o_full0 = p_empty0 + 32;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        int left = (int)blockIdx.y, found = -1, q0 = 0;      // late query tiles (the longest walks) of every head first
        for (int b = rows - 1; b >= row0; --b) {
            const int tiles = (query_start[b + 1] - query_start[b] + tile_q - 1) / tile_q;
            if (left < tiles) { found = b; q0 = (tiles - 1 - left) * tile_q; break; }
            left -= tiles;
        }
        s_row = found; s_q0 = q0;
        mbar_init(q_full, 1);
        for (int s = 0; s < LX_STAGES; ++s) { mbar_init(kv_full0 + 8 * s, 1); mbar_init(kv_empty0 + 8 * s, 3); }
        for (int i = 0; i < 4; ++i) { mbar_init(s_full0 + 8 * i, 1); mbar_init(p_full0 + 8 * i, 4); mbar_init(p_empty0 + 8 * i, 1); }
        for (int g = 0; g < 2; ++g) mbar_init(o_full0 + 8 * g, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 0) {                                          // where the request's gathered rows start
        __syncwarp();
        int before = 0;
        for (int b = row0 + lane; b < s_row; b += 32) before += lx_rows(kv_len[b], query_start[b + 1] - query_start[b], window);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) before += __shfl_xor_sync(0xffffffffu, before, o);
        if (lane == 0) s_at = before;
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "r"(LX_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    const int b = s_row, h = blockIdx.x;
    int tile_lo = 0, t0 = 0, p0 = 0, first_row = 0;
    int g_tiles[2] = {0, 0}, g_qn[2] = {0, 0}, g_hi[2] = {0, 0};
    if (b >= 0) {
        const int nq = query_start[b + 1] - query_start[b], n = kv_len[b];
        t0 = query_start[b] + s_q0;
        p0 = n - nq + s_q0;                                          // position of the CTA's first query
        tile_lo = (window > 0 ? max(0, p0 - window + 1) : 0) / LX_BN;
        first_row = s_at + tile_lo * LX_BN - lx_first(n, nq, window); // gathered row of the walk's first key
#pragma unroll
        for (int g = 0; g < 2; ++g) {
            g_qn[g] = max(0, min(LX_BM, min(nq - s_q0, tile_q) - g * LX_BM));
            g_hi[g] = g_qn[g] ? min(n, p0 + g * LX_BM + g_qn[g]) : 0;
            g_tiles[g] = g_qn[g] ? (g_hi[g] + LX_BN - 1) / LX_BN - tile_lo : 0;
        }
    }
    const int tiles = max(g_tiles[0], g_tiles[1]);

    if (b >= 0 && warp == 0) {
        if (lane == 0) {
            mbar_expect_tx(q_full, 2 * Q_BYTES);
#pragma unroll
            for (int g = 0; g < 2; ++g) {                            // (a group without queries loads rows it never uses)
                const uint32_t dst = q_s + g * Q_BYTES;
#pragma unroll
                for (int i = 0; i < DB; ++i) tma_load_2d(dst + i * 2 * LX_BLOCK, &map_q, q_full, h * q_stride + i * 64, t0 + g * LX_BM);
                tma_load_2d(dst + DB * 2 * LX_BLOCK, &map_qr, q_full, h * qr_stride + qr_at, t0 + g * LX_BM);
            }
            for (int j = 0; j < tiles; ++j) {
                const int s = j % LX_STAGES, row = first_row + j * LX_BN;
                if (!mbar_wait(kv_empty0 + 8 * s, ((j / LX_STAGES) & 1) ^ 1, 1)) break;
                const uint32_t dst = kv_s + s * STAGE;
                mbar_expect_tx(kv_full0 + 8 * s, STAGE);
#pragma unroll
                for (int i = 0; i < DB; ++i) tma_load_2d(dst + i * LX_BLOCK, &map_kv, kv_full0 + 8 * s, h * DIM + i * 64, row);
                tma_load_2d(dst + DB * LX_BLOCK, &map_r, kv_full0 + 8 * s, rank, row);
#pragma unroll
                for (int i = 0; i < VB; ++i) tma_load_2d(dst + (QB + i) * LX_BLOCK, &map_kv, kv_full0 + 8 * s, heads * DIM + h * VDIM + i * 64, row);
            }
        }
    } else if (b >= 0 && (warp == 1 || warp == 10)) {                  // a group's scores S = Q K^T
        if (lane == 0) {
            // kind::f16: D float32, A and B bfloat16; N / 8 at bit 17, M / 16 at bit 24
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LX_BN >> 3) << 17) | ((uint32_t)(LX_BM >> 4) << 24);
            const int g = warp == 1 ? 0 : 1, my_tiles = g_tiles[g];
            bool ok = mbar_wait(q_full, 0, 2);
            for (int j = 0; j < tiles && ok; ++j) {                    // (a group past its own last tile still paces the stages)
                const int s = j % LX_STAGES, gb = g * 2 + (j & 1);
                ok = mbar_wait(kv_full0 + 8 * s, (j / LX_STAGES) & 1, 3);
                if (ok && j < my_tiles) {
                    // S_j overwrites S and P of tile j - 2: wait until P V of that tile has read them
                    if (j >= 2) ok = mbar_wait(p_empty0 + 8 * gb, ((j - 2) >> 1) & 1, 4);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t s_t = tmem + g * 256 + (j & 1) * LX_BN, q_src = q_s + g * Q_BYTES, k_src = kv_s + s * STAGE;
#pragma unroll
                    for (int kk = 0; kk < (DIM + ROT) / 16; ++kk)
                        tc_mma(s_t, tc_smem_desc(q_src + (kk >> 2) * 2 * LX_BLOCK) + (kk & 3) * 2,
                               tc_smem_desc(k_src + (kk >> 2) * LX_BLOCK) + (kk & 3) * 2, idesc, kk != 0);
                    tc_commit(s_full0 + 8 * gb);
                }
                if (ok) tc_commit(kv_empty0 + 8 * s);
            }
        }
    } else if (b >= 0 && warp == 11) {                                // both groups' O += P V
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(VDIM >> 3) << 17) | ((uint32_t)(LX_BM >> 4) << 24);
            bool ok = true;
            for (int j = 0; j < tiles && ok; ++j) {
                const int s = j % LX_STAGES;
                ok = mbar_wait(kv_full0 + 8 * s, (j / LX_STAGES) & 1, 3);
                for (int g = 0; g < 2 && ok; ++g) {
                    if (j >= g_tiles[g]) continue;
                    const int gb = g * 2 + (j & 1);
                    ok = mbar_wait(p_full0 + 8 * gb, (j >> 1) & 1, 5);
                    if (!ok) break;
                    tc_fence_after();
                    const uint32_t v_src = kv_s + s * STAGE + QB * LX_BLOCK, p_t = tmem + g * 256 + (j & 1) * LX_BN;   // P over the first half of its S
#pragma unroll
                    for (int kk = 0; kk < LX_BN / 16; ++kk)           // 16 keys a step: 8 columns along P, 16 rows down V
                        tc_mma_f16_ts(tmem + g * 256 + 2 * LX_BN, p_t + kk * 8, tc_smem_desc_mn(v_src + kk * 16 * 128, LX_BLOCK), idesc, (j | kk) != 0);
                    tc_commit(p_empty0 + 8 * gb);                     // P has been read; O_g holds tile j
                    if (j == g_tiles[g] - 1) tc_commit(o_full0 + 8 * g);
                }
                if (ok) tc_commit(kv_empty0 + 8 * s);
            }
            for (int g = 0; g < 2; ++g)
                if (g_tiles[g] == 0 || !ok) tc_commit(o_full0 + 8 * g);    // (nothing was issued for it, or the walk gave up)
        }
    } else if (b >= 0) {
        const int g = (warp - 2) >> 2;                                // this warp's group of queries
        const int q = warp & 3;                                       // and its quarter of the TMEM lanes = query rows
        const int r = q * 32 + lane, pos = p0 + g * LX_BM + r;        // this thread's query row within the group, and its position
        const int hi = g_hi[g], qn = g_qn[g], my_tiles = g_tiles[g];
        const uint32_t lane_t = tmem + g * 256 + ((uint32_t)(q * 32) << 16), o_t = lane_t + 2 * LX_BN;
        float m_used = -INFINITY, l = 0.f;                            // in log2 units; the maximum may lag by LX_RESCALE
        bool ok = true;
        for (int j = 0; j < my_tiles && ok; ++j) {
            const int gb = g * 2 + (j & 1);
            ok = __all_sync(0xffffffffu, mbar_wait(s_full0 + 8 * gb, (j >> 1) & 1, 6));
            if (!ok) break;
            tc_fence_after();
            uint32_t sr[2][32];
            tc_ld32_nowait(lane_t + (j & 1) * LX_BN, sr[0]);
            tc_ld32_nowait(lane_t + (j & 1) * LX_BN + 32, sr[1]);
            tc_ld_wait();
            const int key0 = (tile_lo + j) * LX_BN;
            if (key0 + LX_BN - 1 > p0 + g * LX_BM || window > 0) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = key0 + c * 32 + i;
                        if (!(key <= pos && key < hi && (window <= 0 || pos - key < window))) sr[c][i] = 0xff800000u;
                    }
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};   // four chains instead of one of 64
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sr[c][i]));
            const float mt = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
            const bool grow = mt > m_used + LX_RESCALE || (m_used == -INFINITY && mt > -INFINITY);
            if (__any_sync(0xffffffffu, grow)) {                      // rescale what is summed (whole warp: the TMEM ops are collective)
                const float m_new = grow ? mt : m_used;
                const float f = m_used == -INFINITY ? 0.f : at_ex2(m_used - m_new);
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(p_empty0 + 8 * (g * 2 + ((j - 1) & 1)), ((j - 1) >> 1) & 1, 7));   // O holds every tile before j
                    tc_fence_after();
                    if (ok) {
#pragma unroll
                        for (int c = 0; c < VDIM / 32; ++c) {
                            uint32_t o[32];
                            tc_ld32(o_t + c * 32, o);
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * f);
                            tc_st32(o_t + c * 32, o);
                        }
                    }
                }
                l *= f;
                m_used = m_new;
            }
            const float off = m_used == -INFINITY ? 0.f : -m_used;
            const uint64_t scale2 = pack2(scale_log2, scale_log2), off2 = pack2(off, off);
            uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};              // four chains of packed sums
            uint32_t pk[32];                                          // 64 weights as bfloat16 pairs
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; i += 2) {
                    float a, d;
                    unpack2(fma2(pack2(__uint_as_float(sr[c][i]), __uint_as_float(sr[c][i + 1])), scale2, off2), a, d);
                    a = at_ex2(a);
                    d = at_ex2(d);
                    sum2[(i >> 1) & 3] = add2(sum2[(i >> 1) & 3], pack2(a, d));
                    __nv_bfloat162 pr = __floats2bfloat162_rn(a, d);
                    pk[c * 16 + i / 2] = *(uint32_t*)&pr;
                }
            float lo, up;
            unpack2(add2(add2(sum2[0], sum2[1]), add2(sum2[2], sum2[3])), lo, up);
            l += lo + up;
            if (!ok) break;
            tc_st32(lane_t + (j & 1) * LX_BN, pk);                    // P over the S it came from: 32 columns of bfloat16 pairs
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full0 + 8 * gb);
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(o_full0 + 8 * g, 0, 9));
        tc_fence_after();
        if (ok && qn > 0) {                                           // (the tensor-memory loads are warp-collective: no lane skips them)
            if (sinks && l > 0.f) l += at_ex2(fmaf(sinks[h], 1.4426950408889634f, -m_used));   // the sink: a weight without a value
            const float inv = l > 0.f ? 1.f / l : 0.f;
            const bool keep = my_tiles > 0 && l != 0.f;              // (a sum that is no number leaves none: O is none then, too)
            bf16* o_row = out + ((size_t)(t0 + g * LX_BM + (r < qn ? r : 0)) * heads + h) * VDIM;
#pragma unroll
            for (int c = 0; c < VDIM / 32; ++c) {
                uint32_t o[32];
                tc_ld32(o_t + c * 32, o);
                if (r < qn) {
#pragma unroll
                    for (int i = 0; i < 32; i += 8) {
                        uint32_t w[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) {
                            const float x = keep ? __uint_as_float(o[i + 2 * e]) * inv : 0.f, y = keep ? __uint_as_float(o[i + 2 * e + 1]) * inv : 0.f;
                            const __nv_bfloat162 pr = __floats2bfloat162_rn(x, y);
                            w[e] = *(const uint32_t*)&pr;
                        }
                        *(uint4*)(o_row + c * 32 + i) = make_uint4(w[0], w[1], w[2], w[3]);
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(LX_TMEM_COLS) : "memory");
    }
}

static int lx_map(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t stride, uint64_t rows, uint32_t box_rows, const char* what) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {stride * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
                                              elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) HB_REFUSE("latent_prompt: cuTensorMapEncodeTiled failed with %d for %s", (int)r, what);
    return 0;
}

HB_DEFINE_STATUS_MIRROR(hb_latent_prompt_status_mirror)
extern "C" int hb_latent_prompt_status(unsigned int* status) {
    HB_CUDA(cudaDeviceSynchronize());
    HB_CUDA(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(unsigned int)));
    const unsigned int zero = 0;
    HB_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(unsigned int)));
    return 0;
}

// Whether the kernel takes these sizes (host only).
extern "C" int hb_latent_prompt_takes(int dim, int rot, int vdim, int rank) {
    return rank >= 16 && rank % 16 == 0 && ((dim == 128 && rot == 64 && vdim == 128) || (dim == 64 && rot == 32 && vdim == 64));
}

extern "C" int hb_latent_gather(void* out, const void* cache, const int32_t* block_table, int table_stride, const int32_t* row_slot,
                                const int32_t* query_start, const int32_t* kv_len, int row0, int rows, int dk, int pages,
                                int page_size, int window, int total, hb_stream stream) {
    if (total <= 0 || rows <= row0) return 0;
    if (dk % 8 || ((uintptr_t)out | (uintptr_t)cache) % 16) HB_REFUSE("latent_gather: rows of %d numbers, or pointers that are not 16-byte aligned", dk);
    latent_gather_kernel<<<(total + 7) / 8, 256, 0, (cudaStream_t)stream>>>(
        (bf16*)out, (const bf16*)cache, block_table, table_stride, row_slot, query_start, kv_len, row0, rows, dk, pages, page_size, window, total);
    HB_LAUNCH_CHECK("latent_gather");
    return 0;
}

template <int DIM, int ROT, int VDIM>
static int lx_launch(void* out, const void* q, int q_ld, const void* qr, const void* rows_kv, const void* lat, const int32_t* query_start,
                     const int32_t* kv_len, int row0, int rows, int q_tiles, int tokens, int heads, int rank, int total, float scale,
                     int window, int tile_q, const float* sinks, cudaStream_t s) {
    CUtensorMap map_q, map_qr, map_kv, map_r;
    const int dk = rank + ROT;
    int rc = lx_map(&map_q, q, (uint64_t)heads * (DIM + ROT), q_ld, tokens, LX_BM, "the queries");
    if (!rc) rc = lx_map(&map_qr, qr, (uint64_t)heads * dk, (uint64_t)heads * dk, tokens, LX_BM, "their rotated parts");
    if (!rc) rc = lx_map(&map_kv, rows_kv, (uint64_t)heads * (DIM + VDIM), (uint64_t)heads * (DIM + VDIM), total, LX_BN, "keys and values");
    if (!rc) rc = lx_map(&map_r, lat, dk, dk, total, LX_BN, "the gathered rows");
    if (rc) return rc;
    constexpr int smem = (2 * (DIM / 64 + 1) * 2 + LX_STAGES * (DIM / 64 + 1 + VDIM / 64)) * LX_BLOCK + 1024;
    auto kernel = latent_prompt_kernel<DIM, ROT, VDIM>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    kernel<<<dim3(heads, q_tiles), LX_THREADS, smem, s>>>(map_q, map_qr, map_kv, map_r, (bf16*)out, query_start, kv_len, row0, rows, heads,
                                                          DIM + ROT, dk, rank, rank, scale * 1.4426950408889634f, window, tile_q, sinks);
    HB_LAUNCH_CHECK("latent_prompt");
    return 0;
}

// Rows row0 .. rows - 1 of the batch; q_tiles is the sum of ceil(queries / tile_q) over them, total the gathered rows' number.
extern "C" int hb_latent_prompt(void* out, const void* q, int q_ld, const void* qa, const void* keys_values, const void* lat,
                                const int32_t* query_start, const int32_t* kv_len, int row0, int rows, int q_tiles, int tokens, int heads,
                                int dim, int rot, int vdim, int rank, int total, float scale, int window, int tile_q,
                                const float* sinks, hb_stream stream) {
    if (rows <= row0 || q_tiles <= 0 || total <= 0) return 0;
    if (!hb_latent_prompt_takes(dim, rot, vdim, rank)) HB_REFUSE("latent_prompt: heads of %d + %d, %d over rank %d do not fit this kernel", dim, rot, vdim, rank);
    if (tile_q != LX_BM && tile_q != 2 * LX_BM) HB_REFUSE("latent_prompt: query tiles of %d (128 or 256)", tile_q);
    if (q_tiles > 65535) HB_REFUSE("latent_prompt: %d query tiles in one step, above 65535", q_tiles);
    if (!(scale > 0.f)) HB_REFUSE("latent_prompt: the score scale must be positive");
    if (q_ld < heads * (dim + rot) || q_ld % 8 || ((uintptr_t)q | (uintptr_t)qa | (uintptr_t)keys_values | (uintptr_t)lat | (uintptr_t)out) % 16)
        HB_REFUSE("latent_prompt: rows of the queries must be a multiple of 8 numbers apart and pointers 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    if (dim == 128)
        return lx_launch<128, 64, 128>(out, q, q_ld, qa, keys_values, lat, query_start, kv_len, row0, rows, q_tiles, tokens, heads, rank, total,
                                       scale, window, tile_q, sinks, s);
    return lx_launch<64, 32, 64>(out, q, q_ld, qa, keys_values, lat, query_start, kv_len, row0, rows, q_tiles, tokens, heads, rank, total,
                                 scale, window, tile_q, sinks, s);
}
