// True 32-bit matrix product: C[M, N] = A[M, K] . W[N, K]^T with float operands and float FMAs
// on the CUDA cores -- no tensor-core mode, no reduced-precision inputs.  It is the matrix
// product of the 32-bit path of the whole model.
//
// out[r] = sum_c W[r, c] * x[c] (integrallis/models, backend-java/.../ops/TensorOps.java:61-63).
// Every output element is the sum, in order, of up to eight chains of FMAs over consecutive parts of
// c = 0..K-1, each in ascending order; the parts follow from N and K alone, so a row's result does not
// depend on how many other rows the call carries, on where the row sits in a tile, on its alignment or on
// which of the kernels below computes it.  (A decode product that need not be row-invariant takes gemv_f32_kernel,
// whose sums run over lanes.)
//
// Bound by shared memory and the FMA pipe together: a lane's 8 x 8 results take 16 operands per column
// of K, 64 bytes through a 128-byte port for the 64 FMAs, both 16 cycles of a multiprocessor per warp.
// 384 rows, 16,384 columns, K 2,048: 1,193 us with 4 x 4 results a thread and element loads, 576 now
// (45 TFLOP/s; the FMA pipes alone would take 346 us); with single FMAs instead of pairs 668; wider results (8 x 16, 12 x 12) lost what they saved to registers.
#include "common.cuh"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kTileM = 64, kTileN = 64, kTileK = 16;

// Any sizes, strides and alignments.
__global__ void __launch_bounds__(256)
gemm_f32_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, float* __restrict__ c,
                int ldc, int m, int n, int k, int part_length) {
    __shared__ float a_tile[kTileK][kTileM + 4];
    __shared__ float w_tile[kTileK][kTileN + 4];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 16 x 16 threads, 4 x 4 outputs each
    const int row0 = blockIdx.y * kTileM, col0 = blockIdx.x * kTileN;
    float acc[4][4] = {}, sum[4][4] = {};
    for (int k0 = 0; k0 < k; k0 += kTileK) {
        if (k0 > 0 && k0 % part_length == 0)  // the next part's chains begin (part_length is a multiple of kTileK)
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    sum[i][j] = k0 == part_length ? acc[i][j] : sum[i][j] + acc[i][j];
                    acc[i][j] = 0.0f;
                }
        // 64 rows x 16 columns of each operand; 256 threads, 4 elements each
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int index = threadIdx.x + i * 256;
            const int r = index / kTileK, kk = index % kTileK;
            const int gr = row0 + r, gc = col0 + r, gk = k0 + kk;
            a_tile[kk][r] = (gr < m && gk < k) ? a[(size_t)gr * lda + gk] : 0.0f;
            w_tile[kk][r] = (gc < n && gk < k) ? w[(size_t)gc * ldw + gk] : 0.0f;
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            float av[4], wv[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) av[i] = a_tile[kk][ty * 4 + i];
#pragma unroll
            for (int j = 0; j < 4; ++j) wv[j] = w_tile[kk][tx * 4 + j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fmaf(av[i], wv[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int gr = row0 + ty * 4 + i;
        if (gr >= m) continue;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int gc = col0 + tx * 4 + j;
            if (gc < n) c[(size_t)gr * ldc + gc] = k > part_length ? sum[i][j] + acc[i][j] : acc[i][j];
        }
    }
}

__device__ __forceinline__ uint64_t twice(float v) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %1};" : "=l"(d) : "f"(v));
    return d;
}
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {  // two float FMAs, each rounded as fmaf rounds
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

__device__ __forceinline__ float low_of(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high_of(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }
__device__ __forceinline__ const float* tiled_part(float* mine, int rank) { return cg::this_cluster().map_shared_rank(mine, rank); }

// Rows of 16-byte pieces.  A block of kWarpsM x kWarpsN warps; a warp is 4 x 8 lanes, a lane holds 4 * kM4 rows x 4 * kN4
// columns, whose fours lie 16 rows (32 columns) apart, so that a four is one 16-byte load from shared memory.  The `parts`
// blocks of a cluster take `part_length` columns of K each; their sums meet in shared memory, added in the parts' order.
template <int kWarpsM, int kWarpsN, int kM4, int kN4>
__global__ void __launch_bounds__(kWarpsM * kWarpsN * 32)
gemm_f32_tiled_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, float* __restrict__ c, int ldc, int m,
                      int n, int k, int tiles_n, int parts, int part_length) {
    constexpr int kThreads = kWarpsM * kWarpsN * 32, kRows = kWarpsM * 16 * kM4, kCols = kWarpsN * 32 * kN4;
    constexpr int kLoadsA = kRows * (kTileK / 4) / kThreads, kLoadsW = kCols * (kTileK / 4) / kThreads;
    static_assert(kLoadsA >= 1 && kLoadsW >= 1 && kRows % 32 == 0 && kCols % 32 == 0, "every thread brings whole pieces");
    // [k][row], the row's bits 3 and 4 turned by k / 4: the eight rows x four pieces that a warp stores at once meet 32 banks
    extern __shared__ __align__(16) float tiled_shared[];
    float* a_tiles = tiled_shared;                          // [2][kTileK][kRows]
    float* w_tiles = tiled_shared + 2 * kTileK * kRows;     // [2][kTileK][kCols]
    const int part = parts > 1 ? (int)cg::this_cluster().block_rank() : 0, tile = blockIdx.x / parts;
    const int row0 = (tile / tiles_n) * kRows, col0 = (tile % tiles_n) * kCols;
    const int k_begin = part * part_length, k_end = min(k, k_begin + part_length);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int my_row = (warp / kWarpsN) * 16 * kM4 + (lane >> 3) * 4, my_col = (warp % kWarpsN) * 32 * kN4 + (lane & 7) * 4;
    uint64_t acc[kM4 * 4][kN4 * 2];
#pragma unroll
    for (int i = 0; i < kM4 * 4; ++i)
#pragma unroll
        for (int j = 0; j < kN4 * 2; ++j) acc[i][j] = 0;
    float4 a_next[kLoadsA], w_next[kLoadsW];
    const int piece = (threadIdx.x & 3) * 4, first = threadIdx.x >> 2;
    auto fetch = [&](int k0) {
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int r = row0 + first + i * (kThreads / 4);
            a_next[i] = (r < m && k0 + piece < k_end) ? __ldg(reinterpret_cast<const float4*>(a + (size_t)r * lda + k0 + piece)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int r = col0 + first + i * (kThreads / 4);
            w_next[i] = (r < n && k0 + piece < k_end) ? __ldg(reinterpret_cast<const float4*>(w + (size_t)r * ldw + k0 + piece)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    };
    auto store = [&](int buffer) {
        const int turn = (piece / 4) << 3;
        float* at = a_tiles + buffer * kTileK * kRows + piece * kRows;
        float* wt = w_tiles + buffer * kTileK * kCols + piece * kCols;
#pragma unroll
        for (int i = 0; i < kLoadsA; ++i) {
            const int r = (first + i * (kThreads / 4)) ^ turn;
            at[r] = a_next[i].x, at[kRows + r] = a_next[i].y, at[2 * kRows + r] = a_next[i].z, at[3 * kRows + r] = a_next[i].w;
        }
#pragma unroll
        for (int i = 0; i < kLoadsW; ++i) {
            const int r = (first + i * (kThreads / 4)) ^ turn;
            wt[r] = w_next[i].x, wt[kCols + r] = w_next[i].y, wt[2 * kCols + r] = w_next[i].z, wt[3 * kCols + r] = w_next[i].w;
        }
    };
    fetch(k_begin);
    store(0);
    __syncthreads();
    const int steps = (k_end - k_begin + kTileK - 1) / kTileK;
    for (int step = 0; step < steps; ++step) {
        const int buffer = step & 1;
        if (step + 1 < steps) fetch(k_begin + (step + 1) * kTileK);
        const float* at = a_tiles + buffer * kTileK * kRows;
        const float* wt = w_tiles + buffer * kTileK * kCols;
#pragma unroll
        for (int kk = 0; kk < kTileK; ++kk) {
            const int turn = (kk / 4) << 3;
            float4 av[kM4];
            ulonglong2 wv[kN4];
#pragma unroll
            for (int i = 0; i < kM4; ++i) av[i] = *reinterpret_cast<const float4*>(at + kk * kRows + ((my_row + 16 * i) ^ turn));
#pragma unroll
            for (int j = 0; j < kN4; ++j) wv[j] = *reinterpret_cast<const ulonglong2*>(wt + kk * kCols + ((my_col + 32 * j) ^ turn));
#pragma unroll
            for (int i = 0; i < kM4; ++i) {
                const uint64_t x[4] = {twice(av[i].x), twice(av[i].y), twice(av[i].z), twice(av[i].w)};
#pragma unroll
                for (int r = 0; r < 4; ++r)
#pragma unroll
                    for (int j = 0; j < kN4; ++j) {
                        acc[4 * i + r][2 * j] = fma_pair(x[r], wv[j].x, acc[4 * i + r][2 * j]);
                        acc[4 * i + r][2 * j + 1] = fma_pair(x[r], wv[j].y, acc[4 * i + r][2 * j + 1]);
                    }
            }
        }
        if (step + 1 < steps) store(buffer ^ 1);  // (the other buffer was last read a step ago, before that step's barrier)
        __syncthreads();
    }
    if (parts == 1) {
#pragma unroll
        for (int i = 0; i < kM4 * 4; ++i) {
            const int r = row0 + my_row + 16 * (i / 4) + i % 4;
            if (r >= m) continue;
#pragma unroll
            for (int j = 0; j < kN4 * 2; ++j) {
                const int to = col0 + my_col + 32 * (j / 2) + 2 * (j % 2);
                if (to < n) c[(size_t)r * ldc + to] = low_of(acc[i][j]);
                if (to + 1 < n) c[(size_t)r * ldc + to + 1] = high_of(acc[i][j]);
            }
        }
        return;
    }
    // this part's sums over the tiles in shared memory (everybody is past the last step), [kRows][kCols]
#pragma unroll
    for (int i = 0; i < kM4 * 4; ++i) {
        const int r = my_row + 16 * (i / 4) + i % 4;
#pragma unroll
        for (int j = 0; j < kN4; ++j)
            *reinterpret_cast<float4*>(tiled_shared + r * kCols + my_col + 32 * j) =
                make_float4(low_of(acc[i][2 * j]), high_of(acc[i][2 * j]), low_of(acc[i][2 * j + 1]), high_of(acc[i][2 * j + 1]));
    }
    cg::this_cluster().sync();
    const int rows_here = kRows / parts;  // (parts is 2, 4 or 8, kRows a multiple of 32)
    for (int i = threadIdx.x; i < rows_here * kCols; i += kThreads) {
        const int r = part * rows_here + i / kCols, col = i % kCols;
        float sum = tiled_part(tiled_shared, 0)[r * kCols + col];
        for (int p = 1; p < parts; ++p) sum += tiled_part(tiled_shared, p)[r * kCols + col];
        if (row0 + r < m && col0 + col < n) c[(size_t)(row0 + r) * ldc + col0 + col] = sum;
    }
    cluster_leave_together();  // the others read this block's sums
}

// Few rows: the weights pass once and bound the product.  A thread owns a column and walks its weights in ascending k; they arrive
// through a ring of kFewDepth stages of kFewStep columns, the rows' own k beside them.  Parts of K as above.
constexpr int kFewRows = 8, kFewColumns = 64, kFewStep = 32, kFewDepth = 4;
constexpr int kFewStride = kFewStep + 4;  // (36 floats: eight lanes' 16-byte loads meet 32 banks)

__device__ __forceinline__ void copy16_async(float* dst, const float* src, bool live) {
    const int bytes = live ? 16 : 0;  // (0: the sixteen bytes are written as zeros and nothing is read)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}

template <int kRows>
__global__ void __launch_bounds__(kFewColumns)
gemm_f32_few_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, float* __restrict__ c, int ldc, int m,
                    int n, int k, int parts, int part_length) {
    constexpr int kPieces = kFewStep / 4, kStage = (kFewColumns + kRows) * kFewStride;
    __shared__ __align__(16) float ring[kFewDepth * kStage];
    __shared__ float sums[kRows][kFewColumns];
    const int part = parts > 1 ? (int)cg::this_cluster().block_rank() : 0;
    const int col0 = (blockIdx.x / parts) * kFewColumns, tid = threadIdx.x;
    const int k_begin = part * part_length, k_end = min(k, k_begin + part_length);
    const int steps = (k_end - k_begin + kFewStep - 1) / kFewStep;
    auto issue = [&](int step) {
        float* stage = ring + (step % kFewDepth) * kStage;
        const int at = (tid % kPieces) * 4, kk = k_begin + step * kFewStep + at;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {  // eight neighbouring threads bring the 128 bytes of a row
            const int r = tid / kPieces + i * (kFewColumns / kPieces);
            const bool live = col0 + r < n && kk < k_end;
            copy16_async(stage + r * kFewStride + at, live ? w + (size_t)(col0 + r) * ldw + kk : w, live);
        }
        static_assert(kFewColumns / kPieces >= kFewRows, "one piece of the rows per thread");
        if (tid / kPieces < kRows) {
            const int r = tid / kPieces;
            const bool live = r < m && kk < k_end;
            copy16_async(stage + (kFewColumns + r) * kFewStride + at, live ? a + (size_t)r * lda + kk : a, live);
        }
    };
    float acc[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) acc[r] = 0.0f;
#pragma unroll
    for (int s = 0; s < kFewDepth - 1; ++s) {
        if (s < steps) issue(s);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    }
    for (int step = 0; step < steps; ++step) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(kFewDepth - 2) : "memory");
        __syncthreads();  // the stage is there for everybody, and everybody is done with the one before
        if (step + kFewDepth - 1 < steps) issue(step + kFewDepth - 1);
        asm volatile("cp.async.commit_group;\n" ::: "memory");
        const float* stage = ring + (step % kFewDepth) * kStage;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const float4 wv = *reinterpret_cast<const float4*>(stage + tid * kFewStride + 4 * i);
#pragma unroll
            for (int r = 0; r < kRows; ++r) {
                const float4 x = *reinterpret_cast<const float4*>(stage + (kFewColumns + r) * kFewStride + 4 * i);
                acc[r] = fmaf(x.x, wv.x, acc[r]);
                acc[r] = fmaf(x.y, wv.y, acc[r]);
                acc[r] = fmaf(x.z, wv.z, acc[r]);
                acc[r] = fmaf(x.w, wv.w, acc[r]);
            }
        }
    }
    if (parts > 1) {
#pragma unroll
        for (int r = 0; r < kRows; ++r) sums[r][tid] = acc[r];
        cg::this_cluster().sync();
        if (part == 0)
#pragma unroll
            for (int r = 0; r < kRows; ++r)
                for (int p = 1; p < parts; ++p) acc[r] += tiled_part(&sums[0][0], p)[r * kFewColumns + tid];
        cluster_leave_together();
        if (part != 0) return;
    }
    if (col0 + tid < n)
#pragma unroll
        for (int r = 0; r < kRows; ++r)
            if (r < m) c[(size_t)r * ldc + col0 + tid] = acc[r];
}

// Few rows (decode): one warp per output column, lanes stride over K, rows kept in registers.
// The per-lane partial sums are combined in a fixed butterfly, so results are reproducible; the
// order differs from the other kernels' sums of chains, which is rounding only.
template <int kRows>
__global__ void __launch_bounds__(256)
gemv_f32_kernel(const float* __restrict__ a, int lda, const float* __restrict__ w, int ldw, float* __restrict__ c,
                int ldc, int m, int n, int k) {
    const int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5, lane = threadIdx.x & 31;
    if (warp >= n) return;
    const float* w_row = w + (size_t)warp * ldw;
    float acc[kRows];
#pragma unroll
    for (int r = 0; r < kRows; ++r) acc[r] = 0.0f;
    for (int kk = lane; kk < k; kk += 32) {
        const float wv = w_row[kk];
#pragma unroll
        for (int r = 0; r < kRows; ++r)
            if (r < m) acc[r] = fmaf(a[(size_t)r * lda + kk], wv, acc[r]);
    }
#pragma unroll
    for (int r = 0; r < kRows; ++r) {
        const float total = warp_sum(acc[r]);
        if (lane == 0 && r < m) c[(size_t)r * ldc + warp] = total;
    }
}

template <typename... Params, typename... Args>
static int launch_parts(void (*kernel)(Params...), unsigned blocks, int threads, int smem, int parts, cudaStream_t stream, Args... args) {
    if (smem > 48 * 1024) {
        cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (status != cudaSuccess) return fail("gemm_f32: cannot reserve %d bytes of shared memory: %s", smem, cudaGetErrorString(status));
    }
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(blocks);
    config.blockDim = dim3(threads);
    config.dynamicSmemBytes = smem;
    config.stream = stream;
    cudaLaunchAttribute attribute[1];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = parts;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    config.attrs = attribute;
    config.numAttrs = parts > 1 ? 1 : 0;
    cudaError_t status = cudaLaunchKernelEx(&config, kernel, args...);
    if (status != cudaSuccess) return fail("gemm_f32: launch failed: %s", cudaGetErrorString(status));
    return check_launch("gemm_f32");
}

template <int kWarpsM, int kWarpsN, int kM4, int kN4>
static int launch_tiled(const float* a, int lda, const float* w, int ldw, float* c, int ldc, int m, int n, int k, int parts, int part_length,
                        cudaStream_t stream) {
    constexpr int kRows = kWarpsM * 16 * kM4, kCols = kWarpsN * 32 * kN4;
    constexpr int tiles_bytes = 2 * kTileK * (kRows + kCols) * (int)sizeof(float), sums_bytes = kRows * kCols * (int)sizeof(float);
    const long long tiles_n = (n + kCols - 1) / kCols, blocks = tiles_n * ((m + kRows - 1) / kRows) * parts;
    if (blocks > 0x7fffffff) return fail("gemm_f32: %d x %d results exceed the grid limit", m, n);
    return launch_parts(gemm_f32_tiled_kernel<kWarpsM, kWarpsN, kM4, kN4>, (unsigned)blocks, kWarpsM * kWarpsN * 32,
                        parts > 1 && sums_bytes > tiles_bytes ? sums_bytes : tiles_bytes, parts, stream, a, lda, w, ldw, c, ldc, m, n, k,
                        (int)tiles_n, parts, part_length);
}

template <int kRows>
static int launch_few(const float* a, int lda, const float* w, int ldw, float* c, int ldc, int m, int n, int k, int parts, int part_length,
                      cudaStream_t stream) {
    return launch_parts(gemm_f32_few_kernel<kRows>, (unsigned)((n + kFewColumns - 1) / kFewColumns * parts), kFewColumns, 0, parts, stream, a, lda,
                        w, ldw, c, ldc, m, n, k, parts, part_length);
}

}  // namespace mb

using namespace mb;

// A: [m, k] with row stride lda; W: [n, k] with row stride ldw; C: [m, n] with row stride ldc.
// `row_invariant` != 0 always takes kernels whose result for a row does not depend on m.
MB_EXPORT int mb_gemm_f32(const float* a, int lda, const float* w, int ldw, float* c, int ldc, int m, int n, int k,
                          int row_invariant, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0) return fail("gemm_f32: k %d must be positive", k);
    if (lda < k || ldw < k || ldc < n) return fail("gemm_f32: row strides (%d, %d, %d) are shorter than the rows (%d, %d, %d)", lda, ldw, ldc, k, k, n);
    if (!row_invariant && m <= 8) {
        const int blocks = (n * 32 + 255) / 256;
        gemv_f32_kernel<8><<<blocks, 256, 0, stream>>>(a, lda, w, ldw, c, ldc, m, n, k);
        return check_launch("gemv_f32");
    }
    // Parts of K, by n and k alone, so that every m and every kernel gives a row the same bits: one chain of 2,048 to 8,192
    // products per result leaves a matrix of few columns with too few of them at work (384 rows, 2,048 columns, K 8,192: 689 us
    // whole, 322 in eight; 2,048 columns, K 2,048: 174 and 94), and shorter chains round less (1.6e-6 and 0.6e-6 from the sums
    // in 64 bits).  Wide matrices gain less (16,384 columns: 596 us whole, 576 in four, 625 in eight).
    int parts = n <= 8192 ? 8 : 4;
    while (parts > 1 && k < 128 * parts) parts /= 2;
    const int part_length = ((k + parts - 1) / parts + kFewStep - 1) / kFewStep * kFewStep;
    if (k % 4 == 0 && lda % 4 == 0 && ldw % 4 == 0 && !((uintptr_t)a & 15) && !((uintptr_t)w & 15)) {
        if (m <= kFewRows) {
            if (m <= 2) return launch_few<2>(a, lda, w, ldw, c, ldc, m, n, k, parts, part_length, stream);
            if (m <= 4) return launch_few<4>(a, lda, w, ldw, c, ldc, m, n, k, parts, part_length, stream);
            return launch_few<8>(a, lda, w, ldw, c, ldc, m, n, k, parts, part_length, stream);
        }
        // Tiles of 64 x 128 where there are two or more per multiprocessor (64 rows, 16,384 columns: 121 us, and 152 in tiles of
        // 32 x 64); else, and where they would be half empty, of 32 x 64 (64 rows, 2,048 columns, K 8,192: 90 us, and 120).
        const long long tiles = (long long)((m + 63) / 64) * ((n + 127) / 128) * parts;
        if (m <= 32 || tiles < 296) return launch_tiled<2, 1, 1, 2>(a, lda, w, ldw, c, ldc, m, n, k, parts, part_length, stream);
        return launch_tiled<2, 2, 2, 2>(a, lda, w, ldw, c, ldc, m, n, k, parts, part_length, stream);
    }
    const dim3 grid((n + kTileN - 1) / kTileN, (m + kTileM - 1) / kTileM);
    if (grid.y > 65535) return fail("gemm_f32: %d rows exceed the grid limit", m);
    gemm_f32_kernel<<<grid, 256, 0, stream>>>(a, lda, w, ldw, c, ldc, m, n, k, part_length);
    return check_launch("gemm_f32");
}
