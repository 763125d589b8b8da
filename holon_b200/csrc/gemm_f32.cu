// out[m, n] = sum_k x[m, k] * w[n, k] in 32-bit on tcgen05 tensor cores: every operand is split into three bfloat16 numbers.
//
// x = x1 + x2 + x3, each the nearest bfloat16 to what the ones before leave (8 + 8 + 8 bits: nothing is left of numbers from 2^-103 on), so
// x w = x1 w1 + (x1 w2 + x2 w1) + (x1 w3 + x2 w2 + x3 w1) up to 2^-26 of |x w|. The six products of 64 columns of k are
// accumulated by tensor cores in 32 bits, the smallest first, and that sum is added to the running one in a register with one
// rounding. Tensor cores cut sums off instead of rounding them, by up to 2^-23 of a step's sum; steps are short so that this does not grow with
// k (up to 512 of k a segment is one step, and it is the whole error).
// Relative error against 64 bits (2-norm), with multiply-adds in up to eight segments before and now: 541 rows, 1,024 of k 2.1e-7 and 0.95e-7;
// 300 rows, 3,072 of k 3.6e-7 and 1.0e-7; operands that are all positive 0.8 to 1.1e-7 and 0.9 to 0.95e-7.
// One order of summation for every output element, a function of k alone: k is cut into up to eight segments of equal length (a multiple
// of 64), each summed in ascending order in steps of 64, and the segments' sums are added pairwise: ((s0 + s1) + (s2 + s3)) + ((s4 + s5) +
// (s6 + s7)). So a row's result does not depend on how many other rows the batch holds, nor on how the work was split.
// A result that is no finite number (an infinity or a NaN among the operands, whose split is none, or an overflow), or so small beside
// its operands that parts below bfloat16's smallest number may be missing from it (GF_TINY), is computed again with multiply-adds on the numbers as they are.
//
// A block takes 128 rows of w (the M side of tcgen05.mma) by up to 96 rows of x. Eight warps read 64 columns of k of both, split them and
// write the planes to shared memory (two stages, 128-byte swizzle); two threads issue the 24 MMAs of a stage each (an MMA keeps its thread for 100 cycles at least, 160 with 96 rows, as far as whole kernels tell); eight warps
// (four in the form for up to 16 rows) read the sums from tensor memory (two buffers) and add them up in registers. A segment's sum waits in tensor memory
// for its partner. Where tiles are few, the blocks of a cluster of SPLIT share a tile's segments and add them through
// distributed shared memory. Many rows are bound by shared memory: 24 MMAs read 168 KB and the planes are written with 84 KB, 2,000 cycles for
// 128 x 96 x 64; few rows by reading w once.
// In us, with multiply-adds and now (1,024 of k if not said): 541 rows, 4,096 columns 113 and 58, 6,144 161 and 78, 1,024 by 3,072 140 and 45; 130 rows,
// 4,096 columns 54 and 19.5; 17 rows, 6,144 37 and 17; 8 rows, 4,096 21 and 11; 2 rows, 151,936 columns 167 and 164; but 2 rows, 6,144 columns 10.4 and 13.8, 1,024 by
// 3,072 7.9 and 13.1: up to four rows pay for a form whose sums do not depend on the rows beside them with the least time of 24 MMAs a step.
// Looking for the largest number and holding the outputs against it takes 2 to 5 % of that (541 rows: 55.3, 74.5 and 42.4 us without).
#include <cooperative_groups.h>

#include "tcgen05.cuh"

namespace cg = cooperative_groups;

#define GF_BM 128                                 // rows of w a tile
#define GF_BK 64                                  // columns of k a step
#define GF_SEGMENTS 8
#define GF_LOADERS 8                              // warps that load and split
#define GF_PLANE (GF_BM * GF_BK * 2)              // bytes of a plane of w

static __host__ __device__ inline int segment_length(int k) {
    return ((k + GF_SEGMENTS - 1) / GF_SEGMENTS + GF_BK - 1) / GF_BK * GF_BK;
}

__device__ __forceinline__ void gf_ld16(uint32_t taddr, float (&v)[16]) {
    uint32_t r[16];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]), "=r"(r[9]),
                   "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr));
    tc_ld_wait();
#pragma unroll
    for (int i = 0; i < 16; ++i) v[i] = __uint_as_float(r[i]);
}
__device__ __forceinline__ void gf_st16(uint32_t taddr, const float (&v)[16]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n"
                 ::"r"(taddr), "f"(v[0]), "f"(v[1]), "f"(v[2]), "f"(v[3]), "f"(v[4]), "f"(v[5]), "f"(v[6]), "f"(v[7]), "f"(v[8]), "f"(v[9]),
                   "f"(v[10]), "f"(v[11]), "f"(v[12]), "f"(v[13]), "f"(v[14]), "f"(v[15])
                 : "memory");
    asm volatile("tcgen05.wait::st.sync.aligned;\n" ::: "memory");
}

// Two numbers into three bfloat16 pairs (packed subtractions: what a loading warp issues is what bounds a step of many rows).
__device__ __forceinline__ void split2(uint64_t v, uint32_t& p1, uint32_t& p2, uint32_t& p3) {
    const uint64_t minus = pack2(-1.f, -1.f);
    float a, b;
    unpack2(v, a, b);
    const __nv_bfloat162 h = __floats2bfloat162_rn(a, b);
    p1 = *(const uint32_t*)&h;
    v = fma2(pack2(__uint_as_float(p1 << 16), __uint_as_float(p1 & 0xffff0000u)), minus, v);
    unpack2(v, a, b);
    const __nv_bfloat162 l = __floats2bfloat162_rn(a, b);
    p2 = *(const uint32_t*)&l;
    v = fma2(pack2(__uint_as_float(p2 << 16), __uint_as_float(p2 & 0xffff0000u)), minus, v);
    unpack2(v, a, b);
    const __nv_bfloat162 t = __floats2bfloat162_rn(a, b);
    p3 = *(const uint32_t*)&t;
}

// Outputs below this times k times the largest number of their rows of x and w (or one) may miss bits: parts of numbers below 2^-103, and parts'
// products, may lie under 2^-126, from where on nothing is taken for granted. That is 2^-125 k of the larger row in all, 2^-24 of such an
// output. It is 1e-27 for 1,024 of k and ordinary rows; only zeros lie below.
#define GF_TINY 0x1p-99f

// An element whose parts gave no finite number or may have lost bits, on the operands themselves.
__device__ __noinline__ float gf_plain(const float* __restrict__ x, const float* __restrict__ w, int k) {
    const int length = segment_length(k);
    float s[GF_SEGMENTS];
#pragma unroll
    for (int q = 0; q < GF_SEGMENTS; ++q) {
        s[q] = 0.f;
        for (int i = q * length; i < min(k, (q + 1) * length); ++i) s[q] = fmaf(x[i], w[i], s[q]);
    }
    return ((s[0] + s[1]) + (s[2] + s[3])) + ((s[4] + s[5]) + (s[6] + s[7]));
}

__device__ __forceinline__ float largest(float a, float b, float c) {   // of three sizes, in one instruction
    asm("max.abs.f32 %0, %0, %1, %2;" : "+f"(a) : "f"(b), "f"(c));
    return a;
}
__device__ __forceinline__ bool gf_infinite(float v) { return !(fabsf(v) <= 3.402823466e38f); }

// Rows row0 .. row1 - 1 of x by this block's columns of the output, which have been written: what the parts of the operands cannot give is made again. Which
// elements those are follows from the element, its row of x and its row of w alone (not from the rows beside them, which only
// decide whether the block looks). `tops` [GF_BM]: room for the largest number of each row of w.
__device__ __noinline__ void gf_repair(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int n, int k, long ldx, long ldo,
                                       int n0, int row0, int row1, float* tops) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5, columns = min(GF_BM, n - n0);
    for (int c = warp; c < columns; c += warps) {
        float top = 0.f;
        for (int i = lane; i < k; i += 32) top = fmaxf(top, fabsf(w[(size_t)(n0 + c) * k + i]));
        top = warp_max(top);
        if (lane == 0) tops[c] = top;
    }
    __syncthreads();
    for (int r = row0 + warp; r < row1; r += warps) {
        const float* xr = x + (size_t)r * ldx;
        float top = 0.f;
        for (int i = lane; i < k; i += 32) top = fmaxf(top, fabsf(xr[i]));
        top = warp_max(top);
        for (int c = lane; c < columns; c += 32) {
            float* o = out + (size_t)r * ldo + n0 + c;
            const float v = *o, other = tops[c];
            const bool small = fabsf(v) < fmaxf(fmaxf(top, other), 1.f) * (GF_TINY * (float)k) && top > 0.f && other > 0.f;
            if (gf_infinite(v) || small) *o = gf_plain(xr, w + (size_t)(n0 + c) * k, k);
        }
    }
}

// ROWS: the most rows of x a tile. rows_x: this launch's (a multiple of 16). ADDERS: warps that add up, four a half of the columns.
template <int ROWS, int ADDERS, int SPLIT, bool VEC>
__global__ void __launch_bounds__(32 * (GF_LOADERS + ADDERS + 2), ROWS <= 16 ? 2 : 1)
gemm_f32_kernel(float* __restrict__ out, const float* __restrict__ x, const float* __restrict__ w, int m, int n, int k, long ldx, long ldo,
                long x_batch, long o_batch, int rows_x) {
    constexpr int SHARE = GF_SEGMENTS / SPLIT, GROUPS = (ROWS / 16 + ADDERS / 4 - 1) / (ADDERS / 4);   // column groups of 16 a warp adds up
    constexpr int LEVELS = SHARE == 8 ? 3 : SHARE == 4 ? 2 : SHARE == 2 ? 1 : 0;                       // sums that wait for their partners
    constexpr uint32_t COLS = ROWS * (2 + LEVELS) <= 32 ? 32 : ROWS * (2 + LEVELS) <= 64 ? 64 : ROWS * (2 + LEVELS) <= 128 ? 128
                            : ROWS * (2 + LEVELS) <= 256 ? 256 : 512;
    extern __shared__ unsigned char smem_raw[];
    const uint32_t base = (smem_addr(smem_raw) + 1023u) & ~1023u;
    float* sums = (float*)(smem_raw + (base - smem_addr(smem_raw)));         // SPLIT > 1, at the end: [rows_x][128] over the stages
    const uint32_t plane_x = rows_x * GF_BK * 2, stage_bytes = 3 * (GF_PLANE + plane_x);
    __shared__ __align__(8) uint64_t bars[8];
    __shared__ uint32_t s_tmem;
    __shared__ float s_top;
    __shared__ float tops[GF_BM];
    const uint32_t full0 = smem_addr(bars), empty0 = full0 + 16, d_full0 = empty0 + 16, d_empty0 = d_full0 + 16;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    x += (size_t)blockIdx.z * x_batch;                                       // blockIdx.z: which of several products (w [batch, n, k])
    out += (size_t)blockIdx.z * o_batch;
    w += (size_t)blockIdx.z * n * k;
    const int n0 = ((int)blockIdx.x / SPLIT) * GF_BM, rank = (int)blockIdx.x % SPLIT, m0 = (int)blockIdx.y * rows_x;
    const int length = segment_length(k), k_first = rank * SHARE * length, k_end = min(k, k_first + SHARE * length);
    const int chunks = k_end > k_first ? (k_end - k_first + GF_BK - 1) / GF_BK : 0, per_segment = length / GF_BK;

    if (threadIdx.x == 0) {
        s_top = 0.f;
        for (int s = 0; s < 2; ++s) {
            mbar_init(full0 + 8 * s, GF_LOADERS); mbar_init(empty0 + 8 * s, 1);
            mbar_init(d_full0 + 8 * s, 1); mbar_init(d_empty0 + 8 * s, ADDERS);
        }
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    if (warp == GF_LOADERS + ADDERS) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(smem_addr(&s_tmem)), "r"(COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = s_tmem;
    if constexpr (SPLIT > 1) {                                               // s_top is there
        __syncwarp();
        cluster_arrive();
    }
    float acc[GROUPS][16];                                                   // (the adders' only)

    if (warp >= ADDERS && warp < ADDERS + GF_LOADERS) {
        // 16 lanes a row of 64 columns, two rows a warp and load, 16 rows a pass of the eight warps
        constexpr int WP = GF_BM / 16, XP = ROWS / 16;
        const int row = (warp - ADDERS) * 2 + (lane >> 4), kk = (lane & 15) * 4;
        float4 v[WP + XP];
        auto fetch = [&](int i, int chunk) {
            const int at = k_first + chunk * GF_BK + kk, r = (i < WP ? n0 : m0) + row + 16 * (i < WP ? i : i - WP);
            const bool there = r < (i < WP ? n : m) && (i < WP || (i - WP) * 16 < rows_x);
            const float* p = (i < WP ? w + (size_t)r * k : x + (size_t)r * ldx) + at;
            if (VEC) return there && at < k_end ? __ldg((const float4*)p) : make_float4(0.f, 0.f, 0.f, 0.f);   // (k and k_end are multiples of 4)
            return make_float4(there && at < k_end ? p[0] : 0.f, there && at + 1 < k_end ? p[1] : 0.f, there && at + 2 < k_end ? p[2] : 0.f,
                               there && at + 3 < k_end ? p[3] : 0.f);
        };
        if (chunks) {
#pragma unroll
            for (int i = 0; i < WP + XP; ++i) v[i] = fetch(i, 0);
        }
        bool ok = true;
        float top = 0.f;                                                     // the largest number (a NaN is none)
        for (int c = 0; c < chunks && ok; ++c) {
            const int s = c & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(empty0 + 8 * s, ((c >> 1) & 1) ^ 1, 1));
            if (!ok) break;
            const uint32_t stage = base + s * stage_bytes;
            const uint32_t within = (uint32_t)((((lane & 15) >> 1) ^ (row & 7)) * 16 + (lane & 1) * 8);   // (row & 7 is the same in every pass)
#pragma unroll
            for (int i = 0; i < WP + XP; ++i) {
                if (i >= WP && (i - WP) * 16 >= rows_x) continue;
                uint32_t p[3][2];
                const uint64_t lo = pack2(v[i].x, v[i].y), hi = pack2(v[i].z, v[i].w);
                split2(lo, p[0][0], p[1][0], p[2][0]);
                split2(hi, p[0][1], p[1][1], p[2][1]);
                top = largest(largest(top, v[i].x, v[i].y), v[i].z, v[i].w);
                const uint32_t at = (i < WP ? stage : stage + 3 * GF_PLANE) + (row + 16 * (i < WP ? i : i - WP)) * 128 + within;
#pragma unroll
                for (int q = 0; q < 3; ++q)
                    asm volatile("st.shared.v2.b32 [%0], {%1, %2};\n" ::"r"(at + q * (i < WP ? GF_PLANE : plane_x)), "r"(p[q][0]), "r"(p[q][1]) : "memory");
                if (c + 1 < chunks) v[i] = fetch(i, c + 1);                  // the next step's numbers are on their way while the rest is split
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(full0 + 8 * s);
        }
        const unsigned most = __reduce_max_sync(0xffffffffu, __float_as_uint(top));   // (numbers from 0 on are ordered as their bits)
        if constexpr (SPLIT > 1) {                                           // in every block of the cluster, once all have set theirs to zero
            __syncwarp();
            cluster_wait();
            if (lane < SPLIT) atomicMax((unsigned*)cg::this_cluster().map_shared_rank(&s_top, lane), most);
        } else if (lane == 0) {
            atomicMax((unsigned*)&s_top, most);
        }
    } else if (warp >= GF_LOADERS + ADDERS) {                                // a stage and buffer each
        if (lane == 0) {
            // kind::f16: D float32 (bit 4), A and B bfloat16 (bits 7, 10), both K-major, N / 8 at bit 17, M / 16 at bit 24
            const uint32_t idesc = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(rows_x >> 3) << 17) | ((uint32_t)(GF_BM >> 4) << 24);
            bool ok = true;
            for (int c = warp - GF_LOADERS - ADDERS; c < chunks && ok; c += 2) {
                const int s = c & 1;
                ok = mbar_wait(d_empty0 + 8 * s, ((c >> 1) & 1) ^ 1, 4);     // the buffer's last sum has been read
                ok = ok && mbar_wait(full0 + 8 * s, (c >> 1) & 1, 2);
                if (!ok) break;
                tc_fence_after();
                const uint32_t stage = base + s * stage_bytes, d = tmem + s * ROWS;
                uint64_t a[3], b[3];
#pragma unroll
                for (int q = 0; q < 3; ++q) { a[q] = tc_smem_desc(stage + q * GF_PLANE); b[q] = tc_smem_desc(stage + 3 * GF_PLANE + q * plane_x); }
#pragma unroll
                for (int q = 0; q < 6; ++q) {                                // w1 x3, w2 x2, w3 x1, w1 x2, w2 x1, w1 x1
                    const int i = q < 3 ? q : q - 3 < 2 ? q - 3 : 0, j = q < 3 ? 2 - q : q < 5 ? 4 - q : 0;
#pragma unroll
                    for (int kk = 0; kk < GF_BK / 16; ++kk) tc_mma(d, a[i] + kk * 2, b[j] + kk * 2, idesc, (q | kk) != 0);
                }
                tc_commit(empty0 + 8 * s);
                tc_commit(d_full0 + 8 * s);
            }
        }
    } else {
        const int half = warp >> 2;                                          // column groups half, half + ADDERS / 4, ...
        const uint32_t lane_t = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        bool ok = true;
        int c = 0;
        for (int q = 0; q < SHARE && ok; ++q) {                              // the segments of this block
#pragma unroll
            for (int g = 0; g < GROUPS; ++g)
#pragma unroll
                for (int i = 0; i < 16; ++i) acc[g][i] = 0.f;
            for (const int until = min(chunks, c + per_segment); c < until; ++c) {
                const int s = c & 1;
                ok = __all_sync(0xffffffffu, mbar_wait(d_full0 + 8 * s, (c >> 1) & 1, 3));
                if (!ok) break;
                tc_fence_after();
#pragma unroll
                for (int g = 0; g < GROUPS; ++g) {
                    const int col = (half + g * (ADDERS / 4)) * 16;
                    if (col < rows_x) {
                        float v[16];
                        gf_ld16(lane_t + s * ROWS + col, v);
#pragma unroll
                        for (int i = 0; i < 16; ++i) acc[g][i] += v[i];
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(d_empty0 + 8 * s);
            }
            if constexpr (LEVELS > 0) {                                      // with its partners, or to wait for them
#pragma unroll
                for (int g = 0; g < GROUPS; ++g) {
                    const int col = (half + g * (ADDERS / 4)) * 16;
                    if (col < rows_x) {
                        int level = 0;
                        for (; (q >> level) & 1; ++level) {
                            float v[16];
                            gf_ld16(lane_t + (2 + level) * ROWS + col, v);
#pragma unroll
                            for (int i = 0; i < 16; ++i) acc[g][i] = v[i] + acc[g][i];
                        }
                        if (q < SHARE - 1) gf_st16(lane_t + (2 + level) * ROWS + col, acc[g]);
                    }
                }
            }
        }
    }
    if constexpr (SPLIT > 1) {
        if (warp < ADDERS || warp >= ADDERS + GF_LOADERS) {
            __syncwarp();
            cluster_wait();
        }
    }
    __syncthreads();                                                         // every stage has been read; alone: s_top is whole
    const float unsafe = GF_TINY * (float)k;
    bool bad = false;
    if constexpr (SPLIT == 1) {
        const int half = warp >> 2, row = (warp & 3) * 32 + lane;
        const float small = fmaxf(s_top, 1.f) * unsafe;
        if (warp < ADDERS) {
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                const int col = (half + g * (ADDERS / 4)) * 16;
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int r = m0 + col + i;
                    if (col >= rows_x || r >= m || n0 + row >= n) continue;
                    out[(size_t)r * ldo + n0 + row] = acc[g][i];
                    bad |= gf_infinite(acc[g][i]) || fabsf(acc[g][i]) < small;
                }
            }
        }
    }
    if constexpr (SPLIT > 1) {                                               // the sums go over the stages
        if (warp < ADDERS) {
            const int half = warp >> 2, row = (warp & 3) * 32 + lane;
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                const int col = (half + g * (ADDERS / 4)) * 16;
                if (col < rows_x)
#pragma unroll
                    for (int i = 0; i < 16; ++i) sums[(col + i) * GF_BM + row] = acc[g][i];
            }
        }
        cg::cluster_group cluster = cg::this_cluster();
        __syncwarp();
        cluster.sync();
        const float small = fmaxf(s_top, 1.f) * unsafe;
        const int quads = rows_x * (GF_BM / 4);                              // this block's share, four columns of the output a thread
        const bool wide = n % 4 == 0 && ldo % 4 == 0 && o_batch % 4 == 0 && (uintptr_t)out % 16 == 0;
        for (int i = rank * (quads / SPLIT) + threadIdx.x; i < (rank + 1) * (quads / SPLIT); i += blockDim.x) {
            const int col = i / (GF_BM / 4), row = i % (GF_BM / 4) * 4, r = m0 + col;
            if (r >= m || n0 + row >= n) continue;
            float4 p[SPLIT];
#pragma unroll
            for (int s = 0; s < SPLIT; ++s) p[s] = *(const float4*)(cluster.map_shared_rank(sums, s) + col * GF_BM + row);
#pragma unroll
            for (int d = 1; d < SPLIT; d *= 2)
#pragma unroll
                for (int s = 0; s < SPLIT; s += 2 * d)
                    p[s] = make_float4(p[s].x + p[s + d].x, p[s].y + p[s + d].y, p[s].z + p[s + d].z, p[s].w + p[s + d].w);
            float v[4] = {p[0].x, p[0].y, p[0].z, p[0].w};
#pragma unroll
            for (int j = 0; j < 4; ++j) bad |= n0 + row + j < n && (gf_infinite(v[j]) || fabsf(v[j]) < small);
            float* o = out + (size_t)r * ldo + n0 + row;
            if (wide) *(float4*)o = make_float4(v[0], v[1], v[2], v[3]);
            else
                for (int j = 0; j < 4; ++j)
                    if (n0 + row + j < n) o[j] = v[j];
        }
        __syncwarp();
        cluster.sync();                                                      // nobody leaves while its sums are being read
    }
    if (__syncthreads_or(bad)) gf_repair(out, x, w, n, k, ldx, ldo, n0, m0 + rank * (rows_x / SPLIT), min(m, m0 + (rank + 1) * (rows_x / SPLIT)), tops);
    tc_fence_before();
    __syncthreads();
    if (warp == GF_LOADERS + ADDERS) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(COLS) : "memory");
    }
}

// ---------------------------------------------------------------- the choice
struct GfArgs { float* out; const float* x; const float* w; int m, n, k, batch; long ldx, ldo, x_batch, o_batch; int rows_x; };

template <int ROWS, int ADDERS, int SPLIT, bool VEC>
static int launch_split(const GfArgs& a, cudaStream_t s) {
    const int smem = 2 * 3 * (GF_PLANE + a.rows_x * GF_BK * 2) + 1024;
    auto kernel = gemm_f32_kernel<ROWS, ADDERS, SPLIT, VEC>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 2 * 3 * (GF_PLANE + ROWS * GF_BK * 2) + 1024));
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((a.n + GF_BM - 1) / GF_BM * SPLIT, (a.m + a.rows_x - 1) / a.rows_x, a.batch);
    config.blockDim = dim3(32 * (GF_LOADERS + ADDERS + 2));
    config.dynamicSmemBytes = smem;
    config.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SPLIT;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = SPLIT > 1 ? 1 : 0;
    HB_CUDA(cudaLaunchKernelEx(&config, kernel, a.out, a.x, a.w, a.m, a.n, a.k, a.ldx, a.ldo, a.x_batch, a.o_batch, a.rows_x));
    return 0;
}

template <int ROWS, int ADDERS>
static int launch_rows(const GfArgs& a, bool vec, int split, cudaStream_t s) {
#define HB_SPLIT(S) (vec ? launch_split<ROWS, ADDERS, S, true>(a, s) : launch_split<ROWS, ADDERS, S, false>(a, s))
    return split == 8 ? HB_SPLIT(8) : split == 4 ? HB_SPLIT(4) : split == 2 ? HB_SPLIT(2) : HB_SPLIT(1);
#undef HB_SPLIT
}

static thread_local int forced_split = 0;
extern "C" int hb_gemm_f32_split(int split) { forced_split = split; return 0; }   // tests: segments shared by so many blocks (0: chosen)

static int launch(const char* what, float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx,
                  long ldo, long x_batch, long o_batch, cudaStream_t s) {
    if (k <= 0) HB_REFUSE("%s: k = %d", what, k);
    if ((m + 63) / 64 > 65535 || batch > 65535)
        HB_REFUSE("%s: %d rows, %d products are above the kernel's limits", what, m, batch);
    const bool vec = (k % 4 == 0) && (ldx % 4 == 0) && (x_batch % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    const bool few = m <= 16;
    const int parts = (m + 95) / 96, rows_x = few ? 16 : ((m + parts - 1) / parts + 15) / 16 * 16;
    // How many blocks share a tile's segments: the launch with the least waves x (steps of 64 columns + what a block costs besides,
    // about four steps, one more for a cluster's sums) wins. Blocks of many rows that walk all of k side by side ask for the same columns of rows
    // whose distance is often a power of two: a step takes them 3.3 to 5 us, shared by two or more 1.8 to 2.2 (541 rows, 6,144 columns: 1,024 of k
    // 119 us by blocks alone, 76 shared; 4,096 of k 581 and 255), so theirs count twice.
    const long tiles = (long)((n + GF_BM - 1) / GF_BM) * ((m + rows_x - 1) / rows_x) * batch, slots = few ? 296 : 148;
    const int steps = segment_length(k) / GF_BK, segments = (k + segment_length(k) - 1) / segment_length(k);
    int split = 1;
    long best = 0;
    for (int c = 1; c <= GF_SEGMENTS; c *= 2) {
        if (c > 1 && c >= 2 * segments) break;
        const int share = GF_SEGMENTS / c, step = c == 1 && !few ? 2 : 1;
        const long cost = (tiles * c + slots - 1) / slots * ((long)min(share, segments) * steps * step + 4 + (c > 1));
        if (c == 1 || cost < best) { best = cost; split = c; }
    }
    if (forced_split) split = forced_split;
    const GfArgs a = {out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, rows_x};
    const int rc = few ? launch_rows<16, 4>(a, vec, split, s) : launch_rows<96, 8>(a, vec, split, s);
    if (rc) return rc;
    HB_LAUNCH_CHECK(what);
    return 0;
}

HB_DEFINE_STATUS_MIRROR(hb_gemm_f32_status_mirror)
extern "C" int hb_gemm_f32_status(unsigned int* status) {
    HB_CUDA(cudaDeviceSynchronize());
    HB_CUDA(cudaMemcpyFromSymbol(status, g_tc_status, sizeof(unsigned int)));
    const unsigned int zero = 0;
    HB_CUDA(cudaMemcpyToSymbol(g_tc_status, &zero, sizeof(unsigned int)));
    return 0;
}

extern "C" int hb_gemm_f32(float* out, const float* x, const float* w, int m, int n, int k, hb_stream stream) {
    if (m == 0 || n == 0) return 0;
    return launch("gemm_f32", out, x, w, m, n, k, 1, k, n, 0, 0, (cudaStream_t)stream);
}

// `batch` products at once, one per head: out[t, b, :] = x[t, b, :] · w[b]ᵀ with w [batch, n, k]; row t of product b
// starts at x + t * ldx + b * x_batch and out + t * ldo + b * o_batch (elements), so heads that lie side by side in
// wider rows are read and written in place.
extern "C" int hb_gemm_f32_heads(float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx,
                                 long x_batch, long ldo, long o_batch, hb_stream stream) {
    if (m == 0 || n == 0 || batch == 0) return 0;
    return launch("gemm_f32_heads", out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, (cudaStream_t)stream);
}
