// The experts' products for prompts on tcgen05 tensor cores by pairs of CTAs, with the weights as the M side.
//
// The rows of all experts lie one after the other (x is gathered into that order first, where it is not in it already). An expert's
// rows are cut into tiles of up to 256, as few as can be and all alike, rounded up to 32, and such a tile is the N side of
// tcgen05.mma (cta_group::2, M 256), whose width is free: 192 rows are one tile of 192 and 312 two of 160, where tiles of 128 rows as the
// M side computed 256 and 384. A pair's tile is those rows by 512 weight rows, as two accumulators of 256 (128 lanes in each CTA's tensor memory): per
// 64-wide k block a CTA loads its 2 x 128 weight rows and half of the tile's rows of x. That is what bounds these products: a
// CTA alone on 128 x 256 asked the L2 for 94 bytes a cycle to keep its tensor pipe busy and got 50; this tile asks for 57 at 192 rows. The
// other bound is reading every expert's weights once. Random choices, with the gather, in us, tiles of 128 rows of x by 256 columns of one CTA and
// this: 2,048 tokens, 6 of 64 experts, 2,048 to 1,408 columns 127 and 109, back 108 and 97; 4 of 32, 2,048 to 3,072 columns 148 and 139, gated
// units of 1,536 150 and 137, of 3,072 from 4,096 545 and 472; 1,024 tokens, gated units of 1,536 125 and 96. (Four epilogue warps
// in place of eight: 201 us for the gated units of 1,536, since both accumulators wait for them.)
// A box may run past its expert's rows or weights (into the next expert's, or past the end, where TMA fills zeros): those
// rows and columns are computed and not stored. Which tiles there are follows from the experts' row counts, which only the device
// knows: every CTA adds them up at its start.
// Gated units (hb_expert_glu_tcgen05, hb_expert_swiglu_tcgen05): an expert's weight is its gate rows, then its up rows; one accumulator holds 256 gate rows, the
// other the 256 up rows beside them, so a thread of the epilogue reads both and applies the gated unit.
// Roles as in gemm_tcgen05_pair.cu: warp 0 of either CTA loads, warp 1 of the leader issues the MMAs, warps 2-9 of either CTA read
// their accumulators: a lane holds one output column, so a warp's store is 64 neighbouring bytes of a row. The two accumulators
// are handed over and back one by one, so the next tile's first MMAs run under this tile's epilogue.
// Every wait is bounded (tcgen05.cuh; status word: hb_experts_tcgen05_status).
#include "tcgen05.cuh"

#define XT_BK 64
#define XT_STAGES 4
#define XT_W_BYTES (128 * XT_BK * 2)              // one accumulator's weight rows of a CTA
#define XT_STAGE_BYTES (3 * XT_W_BYTES)           // two accumulators' weights, up to 128 rows of x
#define XT_MAX_ROWS 256                           // rows of x a tile
#define XT_MAX_EXPERTS 1024
#define XT_THREADS 320                            // a loading, an issuing and eight epilogue warps
#define XT_SMEM (XT_STAGES * XT_STAGE_BYTES + 1024)

__global__ void gather_rows_kernel(bf16* __restrict__ out, const bf16* __restrict__ x, const int32_t* __restrict__ token_of, int k) {
    const size_t r = blockIdx.x;
    const uint4* src = (const uint4*)(x + (size_t)token_of[r] * k);
    uint4* dst = (uint4*)(out + r * k);
    for (int c = threadIdx.x; c < (k >> 3); c += blockDim.x) dst[c] = __ldg(src + c);
}

__device__ __forceinline__ float xt_act(float v, int act) {
    if (act == 1) { v = fmaxf(v, 0.f); return v * v; }
    if (act == 2) return v / (1.f + __expf(-v));
    if (act == 3) return 0.5f * v * (1.f + tanhf(0.7978845608028654f * (v + 0.044715f * v * v * v)));   // gelu, tanh form
    return v;
}

// 1 / (1 + exp(-x)) over exp(-|x|), which is at most one: the divisor lies between one and two, so that its reciprocal needs no care at the
// ends of the range, and one step of Newton's iteration, r + r (1 - d r), takes it to the last bit. (The division written out
// branches, 32 of them one after the other while the next tile waits for the accumulators: gated units of 1,536, 2,048 tokens, 4 of 32 experts
// 152 us in place of 128.)
__device__ __forceinline__ float xt_sigmoid(float x) {
    const float e = __expf(-fabsf(x)), d = 1.f + e, r = __fdividef(1.f, d);
    return (x < 0.f ? e : 1.f) * fmaf(r, fmaf(-d, r, 1.f), r);
}

// What a product's epilogue makes of it: XT_PLAIN an activation; XT_CLAMPED a factor f per row (null: 1), then g = min(f gate, limit),
// u = clamp(f up, +-limit), g sigmoid(alpha g) (u + 1); XT_SWIGLU gate sigmoid(gate) up.
enum XtForm { XT_PLAIN, XT_CLAMPED, XT_SWIGLU };
struct XtGlu {
    const float* row_scale;
    float limit, alpha;
};

// Maps of x with boxes of 128, 64, 32 and 16 rows: half a tile's rows are loaded as the boxes that add up to them.
struct XtMaps { CUtensorMap x[4]; };

struct XtTile { int expert, row, end, width, column; };   // first row, the expert's end, rows a tile (a multiple of 32), column block

// Tile t: expert by expert, the expert's column blocks one after the other, a column block's row tiles side by side (they share
// its weights in the L2).
__device__ __forceinline__ XtTile xt_tile(int t, const int* __restrict__ first, const int32_t* __restrict__ starts, int experts) {
    int lo = 0, hi = experts;                              // first[lo] <= t < first[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (first[mid] <= t) lo = mid; else hi = mid;
    }
    XtTile at;
    at.expert = lo;
    at.row = starts[lo];
    at.end = starts[lo + 1];
    const int rows = at.end - at.row, parts = (rows + XT_MAX_ROWS - 1) / XT_MAX_ROWS, within = t - first[lo];
    at.width = ((rows + parts - 1) / parts + 31) & ~31;
    at.column = within / parts;
    at.row += (within - at.column * parts) * at.width;
    return at;
}

template <int FORM>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(XT_THREADS, 1)
expert_linear_tcgen05_kernel(const __grid_constant__ XtMaps maps, const __grid_constant__ CUtensorMap map_w, bf16* __restrict__ out,
                             const int32_t* __restrict__ starts, int experts, int n, int k, int act, XtGlu glu) {
    constexpr bool GLU = FORM != XT_PLAIN;
    constexpr int SPAN = GLU ? 256 : 512;                  // output columns of a tile
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    __shared__ __align__(8) uint64_t bars[2 * XT_STAGES + 4];
    __shared__ uint32_t s_tmem;
    __shared__ int first[XT_MAX_EXPERTS + 1];              // tiles before each expert's
    const uint32_t full0 = smem_addr(bars), empty0 = full0 + 8 * XT_STAGES;             // full: used in the leader only
    const uint32_t acc_full0 = empty0 + 8 * XT_STAGES, acc_empty0 = acc_full0 + 16;     // acc_empty: used in the leader only
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = cluster_rank();
    const bool leader = rank == 0;
    const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;
    const int kblocks = (k + XT_BK - 1) / XT_BK, blocks_n = (n + SPAN - 1) / SPAN;

    if (threadIdx.x == 0) {
        for (int s = 0; s < XT_STAGES; ++s) { mbar_init(full0 + 8 * s, 1); mbar_init(empty0 + 8 * s, 1); }
        for (int a = 0; a < 2; ++a) { mbar_init(acc_full0 + 8 * a, 1); mbar_init(acc_empty0 + 8 * a, 16); }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == 1) {                                       // the same warp of both CTAs, as the pair's allocation asks
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "r"(512) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;\n" ::: "memory");
    }
    for (int e = threadIdx.x; e < experts; e += blockDim.x)
        first[e + 1] = (starts[e + 1] - starts[e] + XT_MAX_ROWS - 1) / XT_MAX_ROWS * blocks_n;
    __syncthreads();
    if (warp == 0) {
        int sum = 0;
        for (int e0 = 0; e0 < experts; e0 += 32) {
            const int e = e0 + lane;
            int incl = e < experts ? first[e + 1] : 0;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) { const int u = __shfl_up_sync(0xffffffffu, incl, o); if (lane >= o) incl += u; }
            if (e < experts) first[e + 1] = sum + incl;
            sum += __shfl_sync(0xffffffffu, incl, 31);
        }
        if (lane == 0) first[0] = 0;
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();                                        // the partner's barriers exist before anything arrives on them
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    const int tiles = first[experts];

    if (warp == 0) {
        if (lane == 0) {
            int kb_all = 0;                                // k blocks loaded so far, over all tiles
            for (int t = pair; t < tiles; t += pairs) {
                const XtTile at = xt_tile(t, first, starts, experts);
                const int half = at.width >> 1, x0 = at.row + (int)rank * half;
                // (GLU: n is the unit's size, an expert's weight its 2 n rows)
                const int w0 = (GLU ? 2 * at.expert : at.expert) * n + at.column * SPAN + (int)rank * 128, w1 = w0 + (GLU ? n : 256);
                const uint32_t bytes = 2 * (2 * XT_W_BYTES + half * XT_BK * 2);        // of both CTAs
                bool ok = true;
                for (int kb = 0; kb < kblocks && ok; ++kb, ++kb_all) {
                    const int s = kb_all % XT_STAGES;
                    ok = mbar_wait(empty0 + 8 * s, ((kb_all / XT_STAGES) & 1) ^ 1, 1);
                    if (!ok) break;
                    const uint32_t a = base + s * XT_STAGE_BYTES, b = a + 2 * XT_W_BYTES;
                    if (leader) mbar_expect_tx(full0 + 8 * s, bytes);
                    const uint32_t bar = in_cta(full0 + 8 * s, 0);
                    tma_load_2d_pair(a, &map_w, bar, kb * XT_BK, w0);
                    tma_load_2d_pair(a + XT_W_BYTES, &map_w, bar, kb * XT_BK, w1);
                    int r = 0;
#pragma unroll
                    for (int i = 0; i < 4; ++i)
                        if (half & (128 >> i)) { tma_load_2d_pair(b + r * XT_BK * 2, &maps.x[i], bar, kb * XT_BK, x0 + r); r += 128 >> i; }
                }
                if (!ok) break;
            }
        }
    } else if (warp == 1) {
        if (lane == 0 && leader) {
            int kb_all = 0, local = 0;
            bool ok = true;
            for (int t = pair; t < tiles && ok; t += pairs, ++local) {
                const XtTile at = xt_tile(t, first, starts, experts);
                // kind::f16: D float32 (bit 4), A and B bfloat16 (bits 7, 10), both K-major, N / 8 at bit 17, M / 16 at bit 24
                const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(at.width >> 3) << 17) | (16u << 24);
                for (int kb = 0; kb < kblocks && ok; ++kb, ++kb_all) {
                    const int s = kb_all % XT_STAGES;
                    ok = mbar_wait(full0 + 8 * s, (kb_all / XT_STAGES) & 1, 2);
                    if (!ok) break;
                    const uint32_t a = base + s * XT_STAGE_BYTES;
                    const uint64_t da = tc_smem_desc(a), db = tc_smem_desc(a + 2 * XT_W_BYTES);
#pragma unroll
                    for (int acc = 0; acc < 2; ++acc) {
                        if (kb == 0) ok = ok && mbar_wait(acc_empty0 + 8 * acc, (local & 1) ^ 1, 4);   // both epilogues have read it
                        if (!ok) break;
                        tc_fence_after();
#pragma unroll
                        for (int kk = 0; kk < XT_BK / 16; ++kk)
                            tc_mma_pair(tmem + acc * 256, da + (uint64_t)(acc * (XT_W_BYTES >> 4) + kk * 2), db + (uint64_t)(kk * 2), idesc, (kb | kk) != 0);
                        if (kb == kblocks - 1) tc_commit_pair(acc_full0 + 8 * acc);
                    }
                    if (ok) tc_commit_pair(empty0 + 8 * s);
                }
            }
        }
    } else {
        const int q = warp & 3, odd = (warp - 2) >> 2;     // this warp's quarter of the TMEM lanes = columns of the output; every other 32 rows
        const uint32_t acc_empty_leader = in_cta(acc_empty0, 0);
        int local = 0;
        bool ok = true;
        for (int t = pair; t < tiles && ok; t += pairs, ++local) {
            const XtTile at = xt_tile(t, first, starts, experts);
            const int live = min(at.end - at.row, at.width);                 // rows of this tile that exist
            const int col0 = at.column * SPAN + (int)rank * 128 + q * 32 + lane;
            const uint32_t lane_t = tmem + ((uint32_t)(q * 32) << 16);
            auto hand_back = [&](int acc) {
                tc_fence_before();
                __syncwarp();
                if (lane == 0) {
                    mbar_arrive_cluster(acc_empty_leader + 8 * acc);
                    if (GLU) mbar_arrive_cluster(acc_empty_leader + 8);
                }
            };
#pragma unroll
            for (int acc = 0; acc < (GLU ? 1 : 2); ++acc) {
                ok = ok && __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8 * acc, local & 1, 3));
                if (GLU) ok = ok && __all_sync(0xffffffffu, mbar_wait(acc_full0 + 8, local & 1, 3));
                if (!ok) break;
                tc_fence_after();
                const int col = col0 + acc * 256;
                if (32 * odd >= at.width) hand_back(acc);
                for (int c = 32 * odd; c < at.width; c += 64) {
                    uint32_t r[32];
                    float v[32];
                    if constexpr (GLU) {
                        uint32_t r2[32];
                        tc_ld32_nowait(lane_t + c, r);
                        tc_ld32_nowait(lane_t + 256 + c, r2);
                        const float mine = FORM == XT_CLAMPED && glu.row_scale && c + lane < live ? glu.row_scale[at.row + c + lane] : 1.f;
                        tc_ld_wait();
#pragma unroll
                        for (int i = 0; i < 32; ++i) {
                            if (FORM == XT_SWIGLU) {
                                const float g = __uint_as_float(r[i]);
                                v[i] = g * xt_sigmoid(g) * __uint_as_float(r2[i]);
                                continue;
                            }
                            const float f = __shfl_sync(0xffffffffu, mine, i);
                            const float g = fminf(f * __uint_as_float(r[i]), glu.limit);
                            const float u = fminf(fmaxf(f * __uint_as_float(r2[i]), -glu.limit), glu.limit);
                            v[i] = g * xt_sigmoid(glu.alpha * g) * (u + 1.f);
                        }
                    } else {
                        tc_ld32(lane_t + acc * 256 + c, r);
#pragma unroll
                        for (int i = 0; i < 32; ++i) v[i] = xt_act(__uint_as_float(r[i]), act);
                    }
                    if (c + 64 >= at.width) hand_back(acc);    // everything is in registers
                    if (col < n) {
                        bf16* o = out + (size_t)(at.row + c) * n + col;
                        if (c + 32 <= live) {
#pragma unroll
                            for (int i = 0; i < 32; ++i) o[(size_t)i * n] = __float2bfloat16_rn(v[i]);
                        } else {
#pragma unroll
                            for (int i = 0; i < 32; ++i)
                                if (c + i < live) o[(size_t)i * n] = __float2bfloat16_rn(v[i]);
                        }
                    }
                }
            }
        }
    }
    tc_fence_before();
    __syncthreads();
    __syncwarp();
    cluster_sync();                                        // neither CTA leaves, or frees tensor memory, while the other may still use it
    if (warp == 1) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512) : "memory");
    }
}

static int xt_encode_map(CUtensorMap* map, const void* ptr, long rows, int k, int box_rows) {
    const cuuint64_t dims[2] = {(cuuint64_t)k, (cuuint64_t)rows};
    const cuuint64_t strides[1] = {(cuuint64_t)k * 2};
    const cuuint32_t box[2] = {XT_BK, (cuuint32_t)box_rows};
    const cuuint32_t elem[2] = {1, 1};
    const CUresult r = cuTensorMapEncodeTiled(map, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box,
                                              elem, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                                              CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) HB_REFUSE("expert_linear_tcgen05: cuTensorMapEncodeTiled failed with %d (rows %ld, k %d)", (int)r, rows, k);
    return 0;
}

HB_DEFINE_STATUS_MIRROR(hb_experts_tcgen05_status_mirror)
extern "C" int hb_experts_tcgen05_status(unsigned int* status) {
    HB_CUDA(cudaDeviceSynchronize());
    HB_CUDA(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(unsigned int)));
    const unsigned int zero = 0;
    HB_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(unsigned int)));
    return 0;
}

// The shared host half: gathered rows, tensor maps, launch. n: output columns (GLU: the unit's size, an expert's weight having 2 n rows).
template <int FORM>
static int xt_launch(void* out, const void* x, const int32_t* token_of, void* gathered, const void* w, const int32_t* starts,
                     int rows, int experts, int n, int k, int act, XtGlu glu, hb_stream stream) {
    constexpr bool GLU = FORM != XT_PLAIN;
    if (rows == 0 || n == 0) return 0;
    if (k < 8 || k % 8 || n % 8) HB_REFUSE("expert_linear_tcgen05: k = %d and n = %d must be multiples of 8", k, n);
    if (experts < 1 || experts > XT_MAX_EXPERTS) HB_REFUSE("expert_linear_tcgen05: %d experts (1 to %d)", experts, XT_MAX_EXPERTS);
    if (token_of && !gathered) HB_REFUSE("expert_linear_tcgen05: rows that are gathered need room for the gathered copy");
    const void* xs = token_of ? gathered : x;
    if ((((uintptr_t)xs | (uintptr_t)x | (uintptr_t)w | (uintptr_t)out) % 16) != 0) HB_REFUSE("expert_linear_tcgen05: pointers must be 16-byte aligned");
    cudaStream_t s = (cudaStream_t)stream;
    if (token_of) {
        gather_rows_kernel<<<rows, 128, 0, s>>>((bf16*)gathered, (const bf16*)x, token_of, k);
        HB_LAUNCH_CHECK("gather_rows");
    }
    XtMaps maps;
    CUtensorMap map_w;
    for (int i = 0; i < 4; ++i)
        if (int rc = xt_encode_map(&maps.x[i], xs, rows, k, 128 >> i)) return rc;
    if (int rc = xt_encode_map(&map_w, w, (long)experts * n * (GLU ? 2 : 1), k, 128)) return rc;
    HB_CUDA(cudaFuncSetAttribute(expert_linear_tcgen05_kernel<FORM>, cudaFuncAttributeMaxDynamicSharedMemorySize, XT_SMEM));
    static int sms = 0;
    if (sms == 0) {
        int device = 0;
        HB_CUDA(cudaGetDevice(&device));
        HB_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device));
    }
    const int span = GLU ? 256 : 512;
    const long most = (long)(rows / XT_MAX_ROWS + (experts < rows ? experts : rows)) * ((n + span - 1) / span);   // the most tiles any split of the rows has
    const int pairs = (int)(most < sms / 2 ? most : sms / 2);
    expert_linear_tcgen05_kernel<FORM><<<2 * pairs, XT_THREADS, XT_SMEM, s>>>(maps, map_w, (bf16*)out, starts, experts, n, k, act, glu);
    HB_LAUNCH_CHECK("expert_linear_tcgen05");
    return 0;
}

// out [rows, n] = act(x' · w[e]ᵀ) for the rows of expert e (starts [experts + 1]); x' = x gathered by token_of into
// `gathered` [rows, k] (token_of null: x itself, its rows already expert by expert). bfloat16; k and n multiples of 8; pointers
// 16-byte aligned; up to 1,024 experts.
extern "C" int hb_expert_linear_tcgen05(void* out, const void* x, const int32_t* token_of, void* gathered, const void* w,
                                        const int32_t* starts, int rows, int experts, int n, int k, int act, hb_stream stream) {
    return xt_launch<XT_PLAIN>(out, x, token_of, gathered, w, starts, rows, experts, n, k, act, XtGlu{nullptr, 0.f, 0.f}, stream);
}

// out [rows, inter] = silu(gate) up over w [experts, 2 inter, k] (an expert's gate rows, then its up rows).
extern "C" int hb_expert_swiglu_tcgen05(void* out, const void* x, const int32_t* token_of, void* gathered, const void* w,
                                        const int32_t* starts, int rows, int experts, int inter, int k, hb_stream stream) {
    return xt_launch<XT_SWIGLU>(out, x, token_of, gathered, w, starts, rows, experts, inter, k, 0, XtGlu{nullptr, 0.f, 0.f}, stream);
}

// out [rows, inter]: the clamped gated unit over w [experts, 2 inter, k] (an expert's gate rows, then its up rows).
extern "C" int hb_expert_glu_tcgen05(void* out, const void* x, const int32_t* token_of, void* gathered, const void* w,
                                     const int32_t* starts, const float* row_scale, float limit, float alpha,
                                     int rows, int experts, int inter, int k, hb_stream stream) {
    return xt_launch<XT_CLAMPED>(out, x, token_of, gathered, w, starts, rows, experts, inter, k, 0, XtGlu{row_scale, limit, alpha}, stream);
}
