// out[m, n] = sum_k x[m, k] * w[n, k] in true 32-bit on CUDA cores: no tensor cores, no reduced-precision mode.
// One order of summation for every output element, a function of k alone: k is cut into up to eight segments of equal
// length (a multiple of 16, at least 64), each summed in ascending order with fused multiply-adds, and the segments' sums are added in
// ascending order. So a row's result does not depend on how many other rows the batch holds, nor on which of the kernels
// and splits below computed it (and eight shorter sums lose less than one long one).
#include <cooperative_groups.h>

#include "common.cuh"

namespace cg = cooperative_groups;

#define BM 64
#define BN 128
#define BK 16
#define SEGMENTS 8
#define SHORTEST 64                         // terms a segment holds at least: one piece of the kernel for few rows (shorter sums gain nothing)

static __host__ __device__ inline int segment_length(int k) {
    const int share = ((k + SEGMENTS - 1) / SEGMENTS + BK - 1) / BK * BK;
    return share > SHORTEST ? share : SHORTEST;
}

// Two 32-bit multiply-adds in one instruction; each rounds as fmaf does.
__device__ __forceinline__ void fma2(uint64_t& d, uint64_t a, uint64_t b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(d) : "l"(a), "l"(b));
}
__device__ __forceinline__ uint64_t twice(float x) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float2 halves(uint64_t v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}

// ---------------------------------------------------------------- many rows
// Bound by the multiply-adds. 64 x 128 outputs a block of 128 threads, 8 x 8 a thread as packed pairs: 32 packed
// multiply-adds for 4 wide loads from shared memory a step of k (4 x 4 a thread needed 2 for 16 and was bound by them); the
// next 16 columns of k are fetched into registers while these are multiplied. A segment's sum goes to shared memory, so
// that the registers hold one set of sums. Where there are too few tiles for the chip, the blocks of a cluster of SPLIT
// share a tile's segments and add them through distributed shared memory.
// Measured with a 28-layer model of width 1,024 in one pass over 541 rows: its 112 products of 4,096 and 6,144 columns by
// 1,024 take 139 us on average (41 TFLOP/s), those of 1,024 columns by 2,048 and 3,072 109 us. With 64 x 64 tiles and 4 x 4
// outputs a thread this pass and four steps of two rows took 78.7 ms in products, now 18.5. What bounds it: three wavefronts of the
// shared-memory pipe a wide load, 12 for a step of k that multiplies for 16 cycles.
template <bool VEC, int SPLIT>
__global__ void __launch_bounds__(128) gemm_f32_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                       const float* __restrict__ w, int m, int n, int k, long ldx,
                                                       long ldo, long x_batch, long o_batch) {
    extern __shared__ float4 smem4[];
    float (*xs)[BK][BM + 4] = reinterpret_cast<float (*)[BK][BM + 4]>(smem4);
    float (*ws)[BK][BN + 4] = reinterpret_cast<float (*)[BK][BN + 4]>((float*)smem4 + 2 * BK * (BM + 4));
    float* sums = (float*)smem4 + 2 * BK * (BM + BN + 8);               // [SEGMENTS / SPLIT or 1][BM][BN]
    x += (size_t)blockIdx.z * x_batch;                                  // blockIdx.z: which of several products (w [batch, n, k])
    out += (size_t)blockIdx.z * o_batch;
    w += (size_t)blockIdx.z * n * k;
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int m0 = blockIdx.y * BM, n0 = (blockIdx.x / SPLIT) * BN, rank = blockIdx.x % SPLIT;
    const int length = segment_length(k), segments = (k + length - 1) / length;
    constexpr int SHARE = SEGMENTS / SPLIT;
    const int s_first = rank * SHARE, s_last = min(segments, s_first + SHARE);
    const int k_first = s_first * length, k_end = min(k, s_last * length);
    const int steps = k_end > k_first ? (k_end - k_first + BK - 1) / BK : 0, per_segment = length / BK;

    // What this thread loads: 4 neighbouring k (4 lanes a row, so that a warp's load touches 8 lines and not 32: with a row a lane these
    // loads took as much of the L1's bandwidth as all reads of shared memory) of 2 rows of x and 4 of w, 32 rows apart.
    const int lr = tid >> 2, lk = (tid & 3) * 4;
    float xv[2][4], wv[4][4];
    auto fetch4 = [&](float (&v)[4], const float* p, bool there, int kk) {
        if (VEC) {
            const float4 f = there && kk < k ? *(const float4*)(p + kk) : make_float4(0.f, 0.f, 0.f, 0.f);
            v[0] = f.x; v[1] = f.y; v[2] = f.z; v[3] = f.w;
        } else {
#pragma unroll
            for (int j = 0; j < 4; ++j) v[j] = there && kk + j < k ? p[kk + j] : 0.f;
        }
    };
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < 2; ++i) { const int r = m0 + lr + 32 * i; fetch4(xv[i], x + (size_t)(r < m ? r : 0) * ldx, r < m, k0 + lk); }
#pragma unroll
        for (int i = 0; i < 4; ++i) { const int r = n0 + lr + 32 * i; fetch4(wv[i], w + (size_t)(r < n ? r : 0) * k, r < n, k0 + lk); }
    };
    auto stage = [&](int buf) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
#pragma unroll
            for (int i = 0; i < 2; ++i) xs[buf][lk + j][lr + 32 * i] = xv[i][j];
#pragma unroll
            for (int i = 0; i < 4; ++i) ws[buf][lk + j][lr + 32 * i] = wv[i][j];
        }
    };
    const int row = (warp & 1) * 32 + (lane >> 3) * 8, col = (warp >> 1) * 64 + (lane & 7) * 4;   // 8 rows; 4 columns here, 4 at + 32
    uint64_t acc[8][4];
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0;

    if (steps) { fetch(k_first); stage(0); }
    __syncthreads();
    int in_segment = 0, slot = 0;
    for (int step = 0; step < steps; ++step) {
        const int buf = step & 1;
        if (step + 1 < steps) fetch(k_first + (step + 1) * BK);
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const float4 a0 = *(const float4*)&xs[buf][kk][row], a1 = *(const float4*)&xs[buf][kk][row + 4];
            const ulonglong2 b0 = *(const ulonglong2*)&ws[buf][kk][col], b1 = *(const ulonglong2*)&ws[buf][kk][col + 32];
            const float a[8] = {a0.x, a0.y, a0.z, a0.w, a1.x, a1.y, a1.z, a1.w};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                const uint64_t aa = twice(a[i]);
                fma2(acc[i][0], aa, b0.x);
                fma2(acc[i][1], aa, b0.y);
                fma2(acc[i][2], aa, b1.x);
                fma2(acc[i][3], aa, b1.y);
            }
        }
        if (++in_segment == per_segment || step + 1 == steps) {          // the segment's end: its sum to shared memory
            float* at = sums + (SPLIT > 1 ? (size_t)slot * BM * BN : 0);
#pragma unroll
            for (int i = 0; i < 8; ++i)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    float4* p = (float4*)&at[(row + i) * BN + col + 32 * h];
                    const float2 u = halves(acc[i][2 * h]), v = halves(acc[i][2 * h + 1]);
                    float4 s = make_float4(u.x, u.y, v.x, v.y);
                    if (SPLIT == 1 && slot > 0) { const float4 t = *p; s = make_float4(t.x + s.x, t.y + s.y, t.z + s.z, t.w + s.w); }
                    *p = s;
                    acc[i][2 * h] = acc[i][2 * h + 1] = 0;
                }
            in_segment = 0;
            ++slot;
        }
        if (step + 1 < steps) stage(buf ^ 1);
        __syncthreads();
    }
    cg::cluster_group cluster = cg::this_cluster();
    if (SPLIT > 1) cluster.sync();
    constexpr int ROWS = BM / SPLIT;                                     // the tile's rows that this block adds up and writes
    const bool wide = (n % 4 == 0) && (ldo % 4 == 0) && (o_batch % 4 == 0) && ((uintptr_t)out % 16 == 0);
    for (int i = tid; i < ROWS * (BN / 4); i += 128) {
        const int r = rank * ROWS + i / (BN / 4), c = i % (BN / 4) * 4;
        if (m0 + r >= m || n0 + c >= n) continue;
        float4 total = make_float4(0.f, 0.f, 0.f, 0.f);
        if (SPLIT == 1) total = *(const float4*)&sums[r * BN + c];
        else {
            for (int s = 0; s < segments; ++s) {
                const float4 v = *(const float4*)(cluster.map_shared_rank(sums, s / SHARE) + (size_t)(s % SHARE) * BM * BN + r * BN + c);
                total = s ? make_float4(total.x + v.x, total.y + v.y, total.z + v.z, total.w + v.w) : v;
            }
        }
        float* o = out + (size_t)(m0 + r) * ldo + n0 + c;
        if (wide) *(float4*)o = total;
        else {
            const float v[4] = {total.x, total.y, total.z, total.w};
            for (int j = 0; j < 4; ++j)
                if (n0 + c + j < n) o[j] = v[j];
        }
    }
    if (SPLIT > 1) cluster.sync();                                       // nobody leaves while its sums are being read
}

// ---------------------------------------------------------------- few rows
// Bound by reading w once. A block of 256 threads takes 8 columns and all of k: a thread sums one segment of one column
// for a quarter of the rows, over pieces of 64 of each segment that a ring of stages brings by cp.async: three where many
// blocks share an SM, six where there are few blocks (the first five, all of k up to 2,560, are then on their way at once). Two rows, the same
// model's step: 7.2 us for a product of 1,024 columns (10 with three stages), 13.2 on average for the wider ones, the head of 151,936
// columns among them (167 us, 3.7 TB/s); as tiles of 64 rows each was a serial walk over k.
#define FEW_COLS 8
#define FEW_PIECE 64
#define FEW_STRIDE (FEW_PIECE + 4)          // neighbouring (segment, column) rows then lie four banks apart
#define FEW_ROWS 16

__device__ __forceinline__ void copy16(float* dst, const float* src, bool there) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(d), "l"(src), "r"(there ? 16 : 0) : "memory");
}

template <int RT, int FEW_STAGES>           // rows a thread: 4 RT >= m
__global__ void __launch_bounds__(256) gemm_f32_few_kernel(float* __restrict__ out, const float* __restrict__ x,
                                                           const float* __restrict__ w, int m, int n, int k, long ldx,
                                                           long ldo, long x_batch, long o_batch) {
    extern __shared__ float4 smem4[];
    x += (size_t)blockIdx.z * x_batch;
    out += (size_t)blockIdx.z * o_batch;
    w += (size_t)blockIdx.z * n * k;
    const int tid = threadIdx.x, n0 = blockIdx.x * FEW_COLS;
    const int length = segment_length(k), segments = (k + length - 1) / length, pieces = (length + FEW_PIECE - 1) / FEW_PIECE;
    const int stage_floats = SEGMENTS * (FEW_COLS + m) * FEW_STRIDE;
    float* base = (float*)smem4;
    auto load = [&](int piece) {
        float* at = base + (size_t)(piece % FEW_STAGES) * stage_floats;
        const int total = SEGMENTS * (FEW_COLS + m) * (FEW_PIECE / 4);
        for (int i = tid; i < total; i += 256) {
            const int q = i % (FEW_PIECE / 4) * 4, line = i / (FEW_PIECE / 4);      // lines: [segment][column], then [segment][row]
            const bool of_w = line < SEGMENTS * FEW_COLS;
            const int l2 = line - SEGMENTS * FEW_COLS;
            const int s = of_w ? line / FEW_COLS : l2 / m, c = of_w ? n0 + line % FEW_COLS : l2 % m;
            const int in = piece * FEW_PIECE + q, kk = s * length + in;
            const bool there = in < length && kk < k && (!of_w || c < n);
            const float* src = of_w ? w + (size_t)c * k + kk : x + (size_t)c * ldx + kk;
            copy16(at + line * FEW_STRIDE + q, there ? src : x, there);
        }
    };
    const int column = tid & 7, s = (tid >> 3) & 7, group = tid >> 6;
    float acc[RT];
#pragma unroll
    for (int r = 0; r < RT; ++r) acc[r] = 0.f;
#pragma unroll
    for (int p = 0; p < FEW_STAGES - 1; ++p) {
        if (p < pieces) load(p);
        asm volatile("cp.async.commit_group;" ::: "memory");
    }
    const bool busy = group * RT < m && s < segments;
    for (int p = 0; p < pieces; ++p) {
        asm volatile("cp.async.wait_group %0;" ::"n"(FEW_STAGES - 2) : "memory");
        __syncthreads();
        if (p + FEW_STAGES - 1 < pieces) load(p + FEW_STAGES - 1);
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (busy) {
            const float* at = base + (size_t)(p % FEW_STAGES) * stage_floats;
            const float* wl = at + (s * FEW_COLS + column) * FEW_STRIDE;
            const float* xl = at + (SEGMENTS * FEW_COLS + s * m) * FEW_STRIDE;
#pragma unroll 4
            for (int q = 0; q < FEW_PIECE; q += 4) {
                const float4 b = *(const float4*)(wl + q);
#pragma unroll
                for (int r = 0; r < RT; ++r) {
                    const float4 a = *(const float4*)(xl + min(group * RT + r, m - 1) * FEW_STRIDE + q);
                    acc[r] = fmaf(a.w, b.w, fmaf(a.z, b.z, fmaf(a.y, b.y, fmaf(a.x, b.x, acc[r]))));
                }
            }
        }
    }
    __syncthreads();
    float* sums = base;                                                  // [row][segment][column], on the first stage
#pragma unroll
    for (int r = 0; r < RT; ++r)
        if (busy && group * RT + r < m) sums[((group * RT + r) * SEGMENTS + s) * FEW_COLS + column] = acc[r];
    __syncthreads();
    for (int i = tid; i < m * FEW_COLS; i += 256) {
        const int r = i / FEW_COLS, c = i % FEW_COLS;
        if (n0 + c >= n) continue;
        float total = sums[r * SEGMENTS * FEW_COLS + c];
        for (int t = 1; t < segments; ++t) total += sums[(r * SEGMENTS + t) * FEW_COLS + c];
        out[(size_t)r * ldo + n0 + c] = total;
    }
}

// ---------------------------------------------------------------- the choice
template <bool VEC, int SPLIT>
static int launch_tiles(float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx, long ldo,
                        long x_batch, long o_batch, cudaStream_t s) {
    const int smem = (2 * BK * (BM + BN + 8) + (SPLIT > 1 ? SEGMENTS / SPLIT : 1) * BM * BN) * (int)sizeof(float);
    auto kernel = gemm_f32_kernel<VEC, SPLIT>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem));
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((n + BN - 1) / BN * SPLIT, (m + BM - 1) / BM, batch);
    config.blockDim = dim3(128);
    config.dynamicSmemBytes = smem;
    config.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = SPLIT;
    attr[0].val.clusterDim.y = attr[0].val.clusterDim.z = 1;
    config.attrs = attr;
    config.numAttrs = SPLIT > 1 ? 1 : 0;
    HB_CUDA(cudaLaunchKernelEx(&config, kernel, out, x, w, m, n, k, ldx, ldo, x_batch, o_batch));
    return 0;
}

template <int RT, int FEW_STAGES>
static int launch_few_stages(float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx, long ldo,
                      long x_batch, long o_batch, cudaStream_t s) {
    const int smem = FEW_STAGES * SEGMENTS * (FEW_COLS + m) * FEW_STRIDE * (int)sizeof(float);
    auto kernel = gemm_f32_few_kernel<RT, FEW_STAGES>;
    HB_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 FEW_STAGES * SEGMENTS * (FEW_COLS + min(FEW_ROWS, 4 * RT)) * FEW_STRIDE * (int)sizeof(float)));
    kernel<<<dim3((n + FEW_COLS - 1) / FEW_COLS, 1, batch), 256, smem, s>>>(out, x, w, m, n, k, ldx, ldo, x_batch, o_batch);
    return 0;
}

template <int RT>
static int launch_few(float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx, long ldo,
                      long x_batch, long o_batch, cudaStream_t s) {
    const bool deep = (long)((n + FEW_COLS - 1) / FEW_COLS) * batch <= 296 && segment_length(k) > 3 * FEW_PIECE;
    if constexpr (RT == 1)
        if (deep) return launch_few_stages<RT, 6>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s);
    return launch_few_stages<RT, 3>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s);
}

static int launch(const char* what, float* out, const float* x, const float* w, int m, int n, int k, int batch, long ldx,
                  long ldo, long x_batch, long o_batch, cudaStream_t s) {
    if (k <= 0) HB_REFUSE("%s: k = %d", what, k);
    if ((m + BM - 1) / BM > 65535 || batch > 65535)
        HB_REFUSE("%s: %d rows, %d products are above the kernel's limits", what, m, batch);
    const bool vec = (k % 4 == 0) && (ldx % 4 == 0) && (x_batch % 4 == 0) && (((uintptr_t)x | (uintptr_t)w) % 16 == 0);
    int rc;
    // The kernel for few rows reads all of x once per 8 columns: from 9 rows on that is more than the tiles spend on their empty rows,
    // unless there are few columns (k = 1,024 to 3,072, 16 rows: 1,024 columns 17 to 24 us against 24 to 33 as tiles, 6,144 columns 47
    // against 37; 8 rows, 6,144 columns 23).
    if (vec && (m <= FEW_ROWS / 2 || (m <= FEW_ROWS && n <= 2048))) {
        if (m <= 4) rc = launch_few<1>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s);
        else if (m <= 8) rc = launch_few<2>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s);
        else rc = launch_few<4>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s);
    } else {
        // Two blocks an SM keep its multiply-adds busy: with fewer tiles than that, a tile's segments are shared out.
        const long tiles = (long)((n + BN - 1) / BN) * ((m + BM - 1) / BM) * batch;
        const int split = tiles * 8 <= 320 ? 8 : tiles * 4 <= 480 ? 4 : 1;
#define HB_TILES(V, S) launch_tiles<V, S>(out, x, w, m, n, k, batch, ldx, ldo, x_batch, o_batch, s)
        if (vec) rc = split == 8 ? HB_TILES(true, 8) : split == 4 ? HB_TILES(true, 4) : HB_TILES(true, 1);
        else rc = split == 8 ? HB_TILES(false, 8) : split == 4 ? HB_TILES(false, 4) : HB_TILES(false, 1);
#undef HB_TILES
    }
    if (rc) return rc;
    HB_LAUNCH_CHECK(what);
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
