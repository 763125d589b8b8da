// Latent attention of prompt portions in bfloat16 on tcgen05 tensor cores: rank a multiple of 64 up to 256 or of 128 up to
// 512, pages of a multiple of 64 tokens.
//
// All heads read the same cache rows [latent (rank) | rotated key part (rot)], so a request's (token, head) pairs are the M
// side of one problem: its folded queries qa are contiguous rows of rank + rot. A CTA owns 128 of them and walks the
// 64-row tiles of the cache that some of them see:
//   S = Q K^T    tcgen05.mma 128 x 64 x 16 over rank + rot, both operands in shared memory (TMA, 128-byte swizzle, blocks
//                of 64 columns), in two sums: over the blocks that hold output columns of this CTA and over the others, each
//                issued by a warp of its own into 64 columns of tensor memory, two buffers of each;
//   softmax      four warps, one row per thread, which adds the two sums, the running maximum lagging by up to 2^8 (as in attention_tcgen05.cu);
//                the weights go back to tensor memory as bfloat16 pairs, over the first of the sums they came from;
//   O += P C     tcgen05.mma 128 x (rank / VS) x 16, four per tile, P from tensor memory, the same cache rows in shared
//                memory as an MN-major operand.
// An output of 128 x 512 alone would fill tensor memory, so above rank 256 two CTAs (VS = 2, neighbours in the grid) take
// half of the output's columns each and both compute the scores: 1.5 times the multiply-adds, 40 tensor instructions a
// tile and CTA. At rank 512 + 64 the queries take 144 KB of shared memory and leave room for one tile of the cache (72 KB): its
// blocks that hold none of this CTA's output columns are free, and are refilled, as soon as their sum is done, and the
// next tile's begins; the others follow when the weights have been applied. Smaller ranks hold up to three tiles.
// Bound at rank 512 by the chain weights applied -> half of the next tile loaded -> its scores -> softmax, which one tile in shared
// memory does not let overlap. 2,048 tokens, 16 heads, rank 512 + 64: 219 us (one warp for both sums: 234; mma.sync, latent_bf16.cu: 730);
// two prompts of 1,500 and 938 tokens, 16 heads, a window of 1,024: 188 us (187; 519).
// Cache rows past a request's length are zeroed in shared memory before they are used.
// Every mbarrier wait is bounded (tcgen05.cuh).
#include "tcgen05.cuh"

#define LT_BM 128                                 // (token, head) pairs a CTA
#define LT_BN 64                                  // cache rows a tile
#define LT_STAGES 3
#define LT_Q_BLOCK (LT_BM * 128)                  // bytes of a [128 x 64] block of queries
#define LT_K_BLOCK (LT_BN * 128)
#define LT_THREADS 256
#define LT_TMEM_COLS 512                          // buffer i: sums [128 i, 128 i + 64) and [128 i + 64, 128 i + 128); O [256, 256 + rank / VS)
#define LT_O 256
#define LT_RESCALE 8.0f
#define LT_SMEM_MAX 232448

__global__ void __launch_bounds__(LT_THREADS, 1) latent_tcgen05_kernel(
        const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_kv, bf16* __restrict__ out,
        const int32_t* __restrict__ block_table, int table_stride, const int32_t* __restrict__ row_slot,
        const int32_t* __restrict__ query_start, const int32_t* __restrict__ kv_len, int row0, int rows, int heads,
        int rank, int dk, int pages, int page_size, float scale_log2, int window, int stages,
        const float* __restrict__ sinks) {
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    const int blocks = (dk + 63) >> 6, nv = rank / (int)gridDim.x >> 6, v0 = (int)blockIdx.x * nv;   // value blocks [v0, v0 + nv)
    const uint32_t q_s = base, kv_s = q_s + blocks * LT_Q_BLOCK, stage_bytes = blocks * LT_K_BLOCK;
    __shared__ __align__(8) uint64_t bars[1 + 4 * LT_STAGES + 7];
    __shared__ uint32_t s_tmem;
    __shared__ int s_row, s_flat;
    // per stage: the score-only blocks and the value blocks, each full and empty; per S buffer: scores, weights, weights read
    const uint32_t q_full = smem_addr(bars), a_full0 = q_full + 8, a_empty0 = a_full0 + 8 * LT_STAGES;
    const uint32_t v_full0 = a_empty0 + 8 * LT_STAGES, v_empty0 = v_full0 + 8 * LT_STAGES;
    const uint32_t s_full0 = v_empty0 + 8 * LT_STAGES, p_full0 = s_full0 + 16, p_empty0 = p_full0 + 16, o_full = p_empty0 + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;

    if (threadIdx.x == 0) {
        int left = (int)blockIdx.y, found = -1, flat = 0;    // late tiles (the longest walks) first
        for (int b = rows - 1; b >= row0; --b) {
            const int tiles = ((query_start[b + 1] - query_start[b]) * heads + LT_BM - 1) / LT_BM;
            if (left < tiles) { found = b; flat = (tiles - 1 - left) * LT_BM; break; }
            left -= tiles;
        }
        s_row = found; s_flat = flat;
        mbar_init(q_full, 1);
        for (int s = 0; s < LT_STAGES; ++s) {
            mbar_init(a_full0 + 8 * s, 1); mbar_init(a_empty0 + 8 * s, 1);
            mbar_init(v_full0 + 8 * s, 1); mbar_init(v_empty0 + 8 * s, 1);
        }
        for (int i = 0; i < 2; ++i) { mbar_init(s_full0 + 8 * i, 2); mbar_init(p_full0 + 8 * i, 4); mbar_init(p_empty0 + 8 * i, 1); }
        mbar_init(o_full, 1);
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "r"(LT_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;

    const int b = s_row, flat0 = s_flat;
    int n = 0, pos0 = 0, rows_here = 0, tile_lo = 0, tiles = 0, key_hi = 0;
    long flat_global = 0;
    if (b >= 0) {
        const int q0 = query_start[b], nq = query_start[b + 1] - q0;
        n = kv_len[b];
        pos0 = n - nq;                                       // position of the request's first new token
        flat_global = (long)q0 * heads + flat0;
        rows_here = min(LT_BM, nq * heads - flat0);
        key_hi = min(n, pos0 + (flat0 + rows_here - 1) / heads + 1);
        tile_lo = (window > 0 ? max(0, pos0 + flat0 / heads - window + 1) : 0) / LT_BN;
        tiles = max(0, (key_hi + LT_BN - 1) / LT_BN - tile_lo);
    }

    if (b >= 0 && warp == 0) {
        if (lane == 0 && tiles > 0) {
            mbar_expect_tx(q_full, blocks * LT_Q_BLOCK);
            for (int i = 0; i < blocks; ++i) tma_load_2d(q_s + i * LT_Q_BLOCK, &map_q, q_full, i * 64, (int)flat_global);
            const int32_t* table = block_table + (size_t)row_slot[b] * table_stride;
            for (int j = 0; j < tiles; ++j) {
                const int s = j % stages;
                const uint32_t parity = ((j / stages) & 1) ^ 1, dst = kv_s + s * stage_bytes;
                const int key0 = (tile_lo + j) * LT_BN;
                const int page = table[key0 / page_size];
                // of the flattened cache; a page that is none: past its end, where a load reads zeros
                const int row = page < 0 || page >= pages ? pages * page_size : page * page_size + key0 % page_size;
                if (!mbar_wait(a_empty0 + 8 * s, parity, 1)) break;
                mbar_expect_tx(a_full0 + 8 * s, (blocks - nv) * LT_K_BLOCK);
                for (int i = 0; i < blocks; ++i)
                    if (i < v0 || i >= v0 + nv) tma_load_2d(dst + i * LT_K_BLOCK, &map_kv, a_full0 + 8 * s, i * 64, row);
                if (!mbar_wait(v_empty0 + 8 * s, parity, 2)) break;
                mbar_expect_tx(v_full0 + 8 * s, nv * LT_K_BLOCK);
                for (int i = v0; i < v0 + nv; ++i) tma_load_2d(dst + i * LT_K_BLOCK, &map_kv, v_full0 + 8 * s, i * 64, row);
            }
        }
    } else if (b >= 0 && (warp == 1 || warp == 7)) {                          // the scores: blocks without values, blocks with
        // kind::f16, D float32, A and B bfloat16; N / 8 at bit 17, M / 16 at bit 24
        const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(LT_BN >> 3) << 17) | ((uint32_t)(LT_BM >> 4) << 24);
        const bool values = warp == 7;
        const uint32_t full0 = values ? v_full0 : a_full0;
        // (all lanes wait, and agree on how a wait ended: they zero rows together)
        bool ok = tiles > 0 && __all_sync(0xffffffffu, mbar_wait(q_full, 0, 3));
        for (int j = 0; j < tiles && ok; ++j) {
            const int s = j % stages;
            const uint32_t src = kv_s + s * stage_bytes, s_t = tmem + (j & 1) * 2 * LT_BN + (values ? LT_BN : 0);
            const int past = n - (tile_lo + j) * LT_BN;                       // rows of the tile from here on lie past the request's end
            // S_j overwrites the sums and the weights of tile j - 2: wait until those have been applied
            if (j >= 2) ok = __all_sync(0xffffffffu, mbar_wait(p_empty0 + 8 * (j & 1), ((j - 2) >> 1) & 1, 4));
            if (ok) ok = __all_sync(0xffffffffu, mbar_wait(full0 + 8 * s, (j / stages) & 1, 5));
            if (!ok) break;
            if (past < LT_BN) {
                for (int i = 0; i < blocks; ++i)
                    if ((i >= v0 && i < v0 + nv) == values)
                        for (int at = past * 128 + lane * 16; at < LT_K_BLOCK; at += 512)   // (the swizzle stays within a row's 128 bytes)
                            asm volatile("st.shared.v4.b32 [%0], {%1, %1, %1, %1};\n" ::"r"(src + i * LT_K_BLOCK + at), "r"(0) : "memory");
                fence_async_smem();
                __syncwarp();
            }
            if (lane == 0) {
                tc_fence_after();
                uint32_t some = 0;
                for (int i = 0; i < blocks; ++i) {
                    if ((i >= v0 && i < v0 + nv) != values) continue;
                    const int steps = min(4, (dk - i * 64) >> 4);
                    const uint64_t da = tc_smem_desc(q_s + i * LT_Q_BLOCK), db = tc_smem_desc(src + i * LT_K_BLOCK);
                    for (int kk = 0; kk < steps; ++kk) { tc_mma(s_t, da + 2 * kk, db + 2 * kk, idesc, some); some = 1; }
                }
                if (!values) tc_commit(a_empty0 + 8 * s);                     // these blocks have been read
                tc_commit(s_full0 + 8 * (j & 1));
            }
            __syncwarp();
        }
    } else if (b >= 0 && warp == 6) {
        if (lane == 0) {
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | (1u << 16) | ((uint32_t)(nv << 3) << 17) | ((uint32_t)(LT_BM >> 4) << 24);
            const uint32_t o_t = tmem + LT_O;
            bool ok = true;
            for (int j = 0; j < tiles && ok; ++j) {                           // O += P_j C_j
                const int s = j % stages;
                ok = mbar_wait(p_full0 + 8 * (j & 1), (j >> 1) & 1, 6);       // (its scores read the same blocks: they are there)
                if (!ok) break;
                tc_fence_after();
                const uint32_t src = kv_s + s * stage_bytes + v0 * LT_K_BLOCK, p_t = tmem + (j & 1) * 2 * LT_BN;
#pragma unroll
                for (int kk = 0; kk < LT_BN / 16; ++kk)                       // 16 rows a step: 8 columns along P
                    tc_mma_f16_ts(o_t, p_t + kk * 8, tc_smem_desc_mn(src + kk * 16 * 128, LT_K_BLOCK), idesc, (j | kk) != 0);
                tc_commit(p_empty0 + 8 * (j & 1));                            // P has been read; O holds tile j
                tc_commit(v_empty0 + 8 * s);
                if (j == tiles - 1) tc_commit(o_full);
            }
            if (tiles == 0 || !ok) tc_commit(o_full);                         // (nothing was issued, or the walk gave up)
        }
    } else if (b >= 0) {
        const int q = warp & 3, r = q * 32 + lane;                            // this warp's quarter of the TMEM lanes; this thread's row
        const int pos = pos0 + (flat0 + r) / heads;
        const int first_pos = pos0 + flat0 / heads;                           // the tile's first query
        const uint32_t lane_t = tmem + ((uint32_t)(q * 32) << 16), o_t = lane_t + LT_O;
        float m_used = -INFINITY, l = 0.f;                                    // in log2 units; the maximum may lag by LT_RESCALE
        bool ok = true;
        for (int j = 0; j < tiles && ok; ++j) {
            ok = __all_sync(0xffffffffu, mbar_wait(s_full0 + 8 * (j & 1), (j >> 1) & 1, 7));
            if (!ok) break;
            tc_fence_after();
            uint32_t sr[2][32];
            const uint32_t s_t = lane_t + (j & 1) * 2 * LT_BN;
#pragma unroll
            for (int c = 0; c < 2; ++c) {                                     // the two sums of 32 scores
                uint32_t other[32];
                tc_ld32_nowait(s_t + 32 * c, sr[c]);
                tc_ld32_nowait(s_t + LT_BN + 32 * c, other);
                tc_ld_wait();
#pragma unroll
                for (int i = 0; i < 32; ++i) sr[c][i] = __float_as_uint(__uint_as_float(sr[c][i]) + __uint_as_float(other[i]));
            }
            const int key0 = (tile_lo + j) * LT_BN;
            if (key0 + LT_BN - 1 > first_pos || window > 0) {
#pragma unroll
                for (int c = 0; c < 2; ++c)
#pragma unroll
                    for (int i = 0; i < 32; ++i) {
                        const int key = key0 + c * 32 + i;
                        if (!(key <= pos && key < key_hi && (window <= 0 || pos - key < window))) sr[c][i] = 0xff800000u;
                    }
            }
            float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};      // four chains instead of one of 64
#pragma unroll
            for (int c = 0; c < 2; ++c)
#pragma unroll
                for (int i = 0; i < 32; ++i) mx4[i & 3] = fmaxf(mx4[i & 3], __uint_as_float(sr[c][i]));
            const float mt = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * scale_log2;
            const bool grow = mt > m_used + LT_RESCALE || (m_used == -INFINITY && mt > -INFINITY);
            if (__any_sync(0xffffffffu, grow)) {                              // rescale what is summed (whole warp: the TMEM ops are collective)
                const float m_new = grow ? mt : m_used;
                const float f = m_used == -INFINITY ? 0.f : at_ex2(m_used - m_new);
                if (j > 0) {
                    ok = __all_sync(0xffffffffu, mbar_wait(p_empty0 + 8 * ((j - 1) & 1), ((j - 1) >> 1) & 1, 8));   // O holds every tile before j
                    tc_fence_after();
                    if (ok) {
                        for (int c = 0; c < 2 * nv; ++c) {
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
            uint64_t sum2[4] = {0ull, 0ull, 0ull, 0ull};
            uint32_t pk[32];                                                  // 64 weights as bfloat16 pairs
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
            float lo, hi;
            unpack2(add2(add2(sum2[0], sum2[1]), add2(sum2[2], sum2[3])), lo, hi);
            l += lo + hi;
            if (!ok) break;
            tc_st32(s_t, pk);                                                 // P over the first of the sums it came from
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(p_full0 + 8 * (j & 1));
        }
        if (ok) ok = __all_sync(0xffffffffu, mbar_wait(o_full, 0, 9));
        tc_fence_after();
        if (ok) {                                                             // (the tensor-memory loads are warp-collective: no lane skips them)
            if (sinks && l > 0.f) l += at_ex2(fmaf(sinks[(flat0 + r) % heads], 1.4426950408889634f, -m_used));
            const float inv = l > 0.f ? 1.f / l : 0.f;
            const bool keep = tiles > 0 && l != 0.f, mine = r < rows_here;   // (a sum that is no number leaves none: O is none then, too)
            bf16* o_row = out + (size_t)(flat_global + (mine ? r : 0)) * rank + v0 * 64;
            for (int c = 0; c < 2 * nv; ++c) {
                uint32_t o[32];
                tc_ld32(o_t + c * 32, o);
                if (mine) {
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
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(LT_TMEM_COLS) : "memory");
    }
}

static int encode_blocks(CUtensorMap* map, const void* ptr, uint64_t cols, uint64_t rows, uint32_t box_rows, const char* what) {
    const cuuint64_t dims[2] = {cols, rows};
    const cuuint64_t strides[1] = {cols * 2};
    const cuuint32_t box[2] = {64, box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
                                              elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) HB_REFUSE("latent_attention_tcgen05: cuTensorMapEncodeTiled failed with %d for %s", (int)r, what);
    return 0;
}

HB_DEFINE_STATUS_MIRROR(hb_latent_tcgen05_status_mirror)
extern "C" int hb_latent_tcgen05_status(unsigned int* status) {
    HB_CUDA(cudaDeviceSynchronize());
    HB_CUDA(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(unsigned int)));
    const unsigned int zero = 0;
    HB_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(unsigned int)));
    return 0;
}

// Whether the kernel takes these sizes (host only).
extern "C" int hb_latent_tcgen05_takes(int heads, int rank, int rot, int pages, int page_size) {
    if (rank < 64 || rank > 512 || rank % (rank <= 256 ? 64 : 128) || rot < 16 || rot % 16 || page_size % LT_BN || heads < 1) return 0;
    const long blocks = ((long)rank + rot + 63) / 64;
    return blocks * (LT_Q_BLOCK + LT_K_BLOCK) + 1024 <= LT_SMEM_MAX - 1024       // the queries and one tile: up to nine blocks
        && (long)pages * page_size <= 0x7fffffffL;
}

// Rows row0 .. rows - 1 of the batch, which bring `portion` of the step's `tokens` tokens.
extern "C" int hb_latent_attention_tcgen05(void* out, const void* qa, const void* cache, const int32_t* block_table,
                                           int table_stride, const int32_t* row_slot, const int32_t* query_start,
                                           const int32_t* kv_len, int row0, int rows, int tokens, int portion, int heads,
                                           int rank, int rot, int pages, int page_size, float scale, int window,
                                           const float* sinks, hb_stream stream) {
    if (rows <= row0 || portion <= 0) return 0;
    if (!hb_latent_tcgen05_takes(heads, rank, rot, pages, page_size))
        HB_REFUSE("latent_attention_tcgen05: rank %d, rot %d, pages of %d do not fit this kernel", rank, rot, page_size);
    if (!(scale > 0.f)) HB_REFUSE("latent_attention_tcgen05: the score scale must be positive");
    if (((uintptr_t)qa | (uintptr_t)cache | (uintptr_t)out) % 16) HB_REFUSE("latent_attention_tcgen05: pointers must be 16-byte aligned");
    const long tiles = ((long)portion * heads + LT_BM - 1) / LT_BM + (rows - row0);   // the most tiles any cut of the tokens has
    if (tiles > 65535 || (long)tokens * heads > 0x7fffffffL) HB_REFUSE("latent_attention_tcgen05: %ld tiles in one step", tiles);
    const int dk = rank + rot, blocks = (dk + 63) / 64;
    CUtensorMap map_q, map_kv;
    int rc = encode_blocks(&map_q, qa, (uint64_t)dk, (uint64_t)tokens * heads, LT_BM, "the queries");
    if (rc) return rc;
    rc = encode_blocks(&map_kv, cache, (uint64_t)dk, (uint64_t)pages * page_size, LT_BN, "the cache");
    if (rc) return rc;
    const int room = LT_SMEM_MAX - 1024 - 1024 - blocks * LT_Q_BLOCK;         // (1024: alignment; 1024: the static part)
    const int stages = max(1, min(LT_STAGES, room / (blocks * LT_K_BLOCK)));
    const int smem = 1024 + blocks * (LT_Q_BLOCK + stages * LT_K_BLOCK);
    HB_CUDA(cudaFuncSetAttribute(latent_tcgen05_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, LT_SMEM_MAX - 1024));
    latent_tcgen05_kernel<<<dim3(rank > 256 ? 2 : 1, (unsigned)tiles), LT_THREADS, smem, (cudaStream_t)stream>>>(
        map_q, map_kv, (bf16*)out, block_table, table_stride, row_slot, query_start, kv_len, row0, rows, heads, rank, dk,
        pages, page_size, scale * 1.4426950408889634f, window, stages, sinks);
    HB_LAUNCH_CHECK("latent_attention_tcgen05");
    return 0;
}
