// Causal grouped-query attention over a paged cache in plain arithmetic: one warp per (token, head) row, or, for the prompts of
// the 32-bit path with heads of 64 and 128, rows in tiles that share keys and values.
//
// The first takes every size of head (up to 256), float or bfloat16 storage, prompts and single decoded tokens alike.  The two
// are the whole attention of the 32-bit path; the first is the fallback of the bfloat16 path for head sizes its tensor-core
// kernels do not take.
//
// Formula (integrallis/models, backend-java/.../llama/LlamaForwardPass.java:1543-1670 and
// backend-java/.../ops/TensorOps.java:1247-1279): kvHead = head / (heads / kv_heads);
// score_p = dot(q, K[p]) * scale for the visible p; softmax with the maximum subtracted;
// out = sum_p prob_p * V[p].  The softmax here is the running ("online") form of the same sum:
// it keeps a running maximum m and rescales the partial sums when m grows.  All of it in float.
//
// Cache layout of one layer: pool[page][kv_head][page_size][head_dim]; block_table[seq][i] is the
// page that holds positions [i*page_size, (i+1)*page_size) of that sequence.
#include "common.cuh"

#include <math_constants.h>

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kMaxHeadDim = 256;
constexpr int kAccPerLane = kMaxHeadDim / 32;

template <typename T>
__device__ __forceinline__ float dot_row(const float* __restrict__ q_shared, const T* __restrict__ k_row, int head_dim,
                                         bool vector_ok) {
    float sum = 0.0f;
    if (vector_ok) {
        for (int d = 0; d < head_dim; d += 8) {
            float kv[8];
            load8(k_row + d, kv);
#pragma unroll
            for (int i = 0; i < 8; ++i) sum = fmaf(q_shared[d + i], kv[i], sum);
        }
    } else {
        for (int d = 0; d < head_dim; ++d) sum = fmaf(q_shared[d], Num<T>::load(k_row + d), sum);
    }
    return sum;
}

// grid (ceil(max_q_len / warps), heads, sequences); block warps*32.
template <typename T, int kWarps>
__global__ void __launch_bounds__(kWarps * 32)
paged_attention_rows_kernel(const T* __restrict__ q, int q_row_stride, T* __restrict__ out, int out_row_stride,
                            const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                            const int* __restrict__ block_table, int max_blocks, const int* __restrict__ cu_q,
                            const int* __restrict__ kv_lens, int heads, int kv_heads, int head_dim, int page_size,
                            int window, float scale) {
    extern __shared__ float q_shared_all[];  // kWarps * head_dim floats
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seq = blockIdx.z, head = blockIdx.y;
    const int q_begin = cu_q[seq];
    const int q_len = cu_q[seq + 1] - q_begin;
    const int j = blockIdx.x * kWarps + warp;
    if (j >= q_len) return;  // no block-wide barrier below, so a warp may leave alone
    const int kv_len = kv_lens[seq];
    const int pos = kv_len - q_len + j;
    const int first = (window > 0 && pos - window + 1 > 0) ? pos - window + 1 : 0;
    const int kv_head = head / (heads / kv_heads);
    const bool vector_ok = (head_dim % 8) == 0;

    float* q_shared = q_shared_all + warp * head_dim;
    const T* q_row = q + (size_t)(q_begin + j) * q_row_stride + (size_t)head * head_dim;
    for (int d = lane; d < head_dim; d += 32) q_shared[d] = Num<T>::load(q_row + d);
    __syncwarp();

    float acc[kAccPerLane];
#pragma unroll
    for (int i = 0; i < kAccPerLane; ++i) acc[i] = 0.0f;
    float running_max = -CUDART_INF_F, running_sum = 0.0f;
    const int* table = block_table + (size_t)seq * max_blocks;

    for (int chunk = first - (first % 32); chunk <= pos; chunk += 32) {
        // page_size is a multiple of 32, so a chunk of 32 positions lies in one page
        const size_t page = table[chunk / page_size];
        const size_t base = ((page * kv_heads + kv_head) * page_size + (chunk % page_size)) * head_dim;
        const int p = chunk + lane;
        const bool visible = p >= first && p <= pos;
        float score = -CUDART_INF_F;
        if (visible) score = dot_row<T>(q_shared, k_pool + base + (size_t)lane * head_dim, head_dim, vector_ok) * scale;
        const float chunk_max = warp_max(score);
        const float new_max = fmaxf(running_max, chunk_max);  // finite: position `pos` is visible in the last chunk,
                                                              // and earlier chunks hold at least one visible key
        const float e = visible ? expf(score - new_max) : 0.0f;
        const float correction = expf(running_max - new_max);  // exp(-inf) = 0 on the first chunk
        running_sum = running_sum * correction + warp_sum(e);
        running_max = new_max;
#pragma unroll
        for (int i = 0; i < kAccPerLane; ++i) acc[i] *= correction;
        const int last = (pos - chunk < 31) ? pos - chunk : 31;
        const int begin = first > chunk ? first - chunk : 0;
        for (int jj = begin; jj <= last; ++jj) {
            const float prob = __shfl_sync(0xffffffffu, e, jj);
            const T* v_row = v_pool + base + (size_t)jj * head_dim;
#pragma unroll
            for (int i = 0; i < kAccPerLane; ++i) {
                const int d = lane + 32 * i;
                if (d < head_dim) acc[i] = fmaf(prob, Num<T>::load(v_row + d), acc[i]);
            }
        }
    }
    const float inv_sum = 1.0f / running_sum;
    T* out_row = out + (size_t)(q_begin + j) * out_row_stride + (size_t)head * head_dim;
#pragma unroll
    for (int i = 0; i < kAccPerLane; ++i) {
        const int d = lane + 32 * i;
        if (d < head_dim) Num<T>::store(out_row + d, acc[i] * inv_sum);
    }
}

// The same for the prompts of the 32-bit path, several rows at a time: the rows of a block (16: the query heads of one kv head, token
// after token) share their keys and values through shared memory, a warp's four rows every key and value that a lane has read.  A row's
// operations and their order are those of the kernel above -- 32 positions a chunk, a lane per key, the running sum rescaled once a
// chunk -- so that a token's result is the same bits whether it came with a prompt or alone.
// Bound by the chunks of the longest rows one after another, each a chain of a dot product, two reductions over lanes and a pass over the
// values.  32 heads of 64 over 8 kv heads, prompts of 170 and 131 tokens: 113 us with a warp a row, 28.5 now (40.9 in tiles of 32
// rows with eight a warp, 35.1 with four a warp, 29.6 in tiles of 16 with two); 400 tokens 348 and 62; 30, 20 and 10 tokens 14.7 and 9.5.
constexpr int kTileRows = 16, kWarpRows = 4, kTileThreads = 32 * kTileRows / kWarpRows;

template <int HD>
struct RowTiles {
    static constexpr int kKeyRow = HD + 4;  // floats: eight lanes' 16-byte loads, a row each, meet 32 banks
    static constexpr int kStageFloats = 32 * kKeyRow + 32 * HD;
    static constexpr int kBytes = (2 * kStageFloats + kTileRows * HD + kTileRows * 32) * (int)sizeof(float);
};

__device__ __forceinline__ void copy16(float* to, const float* from) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(to)), "l"(from) : "memory");
}

// grid (ceil(max_q_len * heads per kv head / 16), kv_heads, sequences).
template <int HD>
__global__ void __launch_bounds__(kTileThreads)
paged_attention_row_tiles_kernel(const float* __restrict__ q, int q_row_stride, float* __restrict__ out, int out_row_stride,
                                 const float* __restrict__ k_pool, const float* __restrict__ v_pool, const int* __restrict__ block_table,
                                 int max_blocks, const int* __restrict__ cu_q, const int* __restrict__ kv_lens, int heads, int kv_heads,
                                 int page_size, int window, float scale) {
    using Tiles = RowTiles<HD>;
    extern __shared__ __align__(16) float tile_smem[];
    float* q_rows = tile_smem + 2 * Tiles::kStageFloats;            // [16][HD]
    float* weights = q_rows + kTileRows * HD;                       // [16][32]
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int seq = blockIdx.z, kv_head = blockIdx.y, group = heads / kv_heads;
    const int q_begin = cu_q[seq], q_len = cu_q[seq + 1] - q_begin;
    const int row0 = blockIdx.x * kTileRows, rows = min(kTileRows, q_len * group - row0);  // row: token * group + head of the group
    if (rows <= 0) return;
    const int kv_len = kv_lens[seq], pos0 = kv_len - q_len;  // the position of the sequence's first new token
    auto first_of = [&](int pos) { return window > 0 && pos - window + 1 > 0 ? pos - window + 1 : 0; };
    const int block_last = pos0 + (row0 + rows - 1) / group, block_first = first_of(pos0 + row0 / group);
    const int* table = block_table + (size_t)seq * max_blocks;

    auto fetch = [&](int chunk, int stage) {  // 32 positions of one page
        const size_t base = (((size_t)table[chunk / page_size] * kv_heads + kv_head) * page_size + chunk % page_size) * HD;
        float* keys = tile_smem + stage * Tiles::kStageFloats;
        float* values = keys + 32 * Tiles::kKeyRow;
#pragma unroll
        for (int i = threadIdx.x; i < 32 * HD / 4; i += kTileThreads) {
            copy16(keys + i / (HD / 4) * Tiles::kKeyRow + i % (HD / 4) * 4, k_pool + base + 4 * i);
            copy16(values + 4 * i, v_pool + base + 4 * i);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int chunk_begin = block_first - block_first % 32;
    fetch(chunk_begin, 0);
    for (int i = threadIdx.x; i < rows * (HD / 4); i += kTileThreads) {
        const int r = row0 + i / (HD / 4), at = i % (HD / 4) * 4;
        *reinterpret_cast<float4*>(q_rows + i * 4) =
            *reinterpret_cast<const float4*>(q + (size_t)(q_begin + r / group) * q_row_stride + (size_t)(kv_head * group + r % group) * HD + at);
    }
    const int mine = warp * kWarpRows, live = min(kWarpRows, rows - mine);  // (of a warp beyond the last row: none)
    const float* my_q = q_rows + mine * HD;
    float* my_weights = weights + mine * 32;
    int pos[kWarpRows];
#pragma unroll
    for (int r = 0; r < kWarpRows; ++r) pos[r] = r < live ? pos0 + (row0 + mine + r) / group : -1;
    float acc[kWarpRows][HD / 32], running_max[kWarpRows], running_sum[kWarpRows];
#pragma unroll
    for (int r = 0; r < kWarpRows; ++r) {
        running_max[r] = -CUDART_INF_F, running_sum[r] = 0.0f;
#pragma unroll
        for (int i = 0; i < HD / 32; ++i) acc[r][i] = 0.0f;
    }

    int stage = 0;
    for (int chunk = chunk_begin; chunk <= block_last; chunk += 32, stage ^= 1) {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
        __syncthreads();  // the chunk is there for everybody, and everybody is done with the one before
        if (chunk + 32 <= block_last) fetch(chunk + 32, stage ^ 1);
        const float* keys = tile_smem + stage * Tiles::kStageFloats;
        const float* values = keys + 32 * Tiles::kKeyRow;
        float score[kWarpRows];
#pragma unroll
        for (int r = 0; r < kWarpRows; ++r) score[r] = 0.0f;
#pragma unroll 4
        for (int d = 0; d < HD; d += 4) {
            const float4 k = *reinterpret_cast<const float4*>(keys + lane * Tiles::kKeyRow + d);
#pragma unroll
            for (int r = 0; r < kWarpRows; ++r) {  // (rows that are not there: what lies behind the others, unused)
                const float4 x = *reinterpret_cast<const float4*>(my_q + r * HD + d);
                score[r] = fmaf(x.x, k.x, score[r]);
                score[r] = fmaf(x.y, k.y, score[r]);
                score[r] = fmaf(x.z, k.z, score[r]);
                score[r] = fmaf(x.w, k.w, score[r]);
            }
        }
        // whether every row sees all of the chunk, and rows that see something of it
        bool whole = live == kWarpRows;
        uint32_t sees = 0;
        const int p = chunk + lane;
#pragma unroll
        for (int r = 0; r < kWarpRows; ++r) {
            const int first = first_of(pos[r]);
            whole = whole && first <= chunk && chunk + 31 <= pos[r];
            if (chunk > pos[r] || chunk + 31 < first) continue;  // (the same for all lanes; of rows that are not there: always)
            sees |= 1u << r;
            const bool visible = p >= first && p <= pos[r];
            const float s = visible ? score[r] * scale : -CUDART_INF_F;
            const float new_max = fmaxf(running_max[r], warp_max(s));
            const float e = visible ? expf(s - new_max) : 0.0f;
            const float correction = expf(running_max[r] - new_max);
            running_sum[r] = running_sum[r] * correction + warp_sum(e);
            running_max[r] = new_max;
#pragma unroll
            for (int i = 0; i < HD / 32; ++i) acc[r][i] *= correction;
            my_weights[r * 32 + lane] = e;
        }
        __syncwarp();
        if (whole) {
#pragma unroll 2
            for (int j = 0; j < 32; j += 4) {
                float v[4][HD / 32];
#pragma unroll
                for (int e = 0; e < 4; ++e)
#pragma unroll
                    for (int i = 0; i < HD / 32; ++i) v[e][i] = values[(j + e) * HD + lane + 32 * i];
#pragma unroll
                for (int r = 0; r < kWarpRows; ++r) {
                    const float4 w = *reinterpret_cast<const float4*>(my_weights + r * 32 + j);
#pragma unroll
                    for (int i = 0; i < HD / 32; ++i) {
                        acc[r][i] = fmaf(w.x, v[0][i], acc[r][i]);
                        acc[r][i] = fmaf(w.y, v[1][i], acc[r][i]);
                        acc[r][i] = fmaf(w.z, v[2][i], acc[r][i]);
                        acc[r][i] = fmaf(w.w, v[3][i], acc[r][i]);
                    }
                }
            }
        } else {  // an end of a row's positions lies here: what it does not see must not be multiplied, not even by zero
#pragma unroll
            for (int r = 0; r < kWarpRows; ++r) {
                if ((sees >> r & 1) == 0) continue;
                const int begin = max(0, first_of(pos[r]) - chunk), last = min(31, pos[r] - chunk);
#pragma unroll 4
                for (int j = begin; j <= last; ++j) {
                    const float w = my_weights[r * 32 + j];
#pragma unroll
                    for (int i = 0; i < HD / 32; ++i) acc[r][i] = fmaf(w, values[j * HD + lane + 32 * i], acc[r][i]);
                }
            }
        }
        __syncwarp();  // the weights have been read
    }
#pragma unroll
    for (int r = 0; r < kWarpRows; ++r)
        if (r < live) {
            const int row = row0 + mine + r;
            const float inv_sum = 1.0f / running_sum[r];
            float* to = out + (size_t)(q_begin + row / group) * out_row_stride + (size_t)(kv_head * group + row % group) * HD;
#pragma unroll
            for (int i = 0; i < HD / 32; ++i) to[lane + 32 * i] = acc[r][i] * inv_sum;
        }
}

template <int HD>
static int launch_row_tiles(const float* q, int q_row_stride, float* out, int out_row_stride, const float* k_pool, const float* v_pool,
                            const int* block_table, int max_blocks, const int* cu_q, const int* kv_lens, int sequences, long long rows,
                            int heads, int kv_heads, int page_size, int window, float scale, cudaStream_t stream) {
    static DeviceSet devices{0};
    if (int status = reserve_shared("paged_attention_rows", paged_attention_row_tiles_kernel<HD>, RowTiles<HD>::kBytes, devices)) return status;
    const dim3 grid((unsigned)((rows + kTileRows - 1) / kTileRows), kv_heads, sequences);
    paged_attention_row_tiles_kernel<HD><<<grid, kTileThreads, RowTiles<HD>::kBytes, stream>>>(
        q, q_row_stride, out, out_row_stride, k_pool, v_pool, block_table, max_blocks, cu_q, kv_lens, heads, kv_heads, page_size, window, scale);
    return check_launch("paged_attention_rows");
}

}  // namespace mb

using namespace mb;

// q: rows of `heads` heads (row stride in elements), out likewise.  cu_q[sequences + 1] are the
// first rows of each sequence's new tokens; kv_lens[sequences] the cache lengths including them.
MB_EXPORT int mb_paged_attention_rows(const void* q, int q_row_stride, void* out, int out_row_stride, int dtype,
                                      const void* k_pool, const void* v_pool, const int* block_table, int max_blocks,
                                      const int* cu_q, const int* kv_lens, int sequences, int max_q_len, int heads,
                                      int kv_heads, int head_dim, int page_size, int window, float scale,
                                      cudaStream_t stream) {
    if (sequences <= 0 || max_q_len <= 0) return 0;
    if (head_dim <= 0 || head_dim > kMaxHeadDim) return fail("paged_attention_rows: head_dim %d is outside 1..%d", head_dim, kMaxHeadDim);
    if (kv_heads <= 0 || heads % kv_heads) return fail("paged_attention_rows: %d heads are no multiple of %d kv heads", heads, kv_heads);
    if (page_size <= 0 || page_size % 32) return fail("paged_attention_rows: page_size %d must be a multiple of 32", page_size);
    if (sequences > 65535) return fail("paged_attention_rows: %d sequences exceed the grid limit 65535", sequences);
    if (heads > 65535) return fail("paged_attention_rows: %d heads exceed the grid limit 65535", heads);
    // Prompts of floats in rows of 16-byte pieces go in tiles; single tokens would leave all but a group's rows of a tile empty.  (Where
    // there are two to five positions in all a warp a row is the faster, by 0.3 to 1.2 of 5 us; with 40 tiles are, 14.5 -> 8.5.  Nobody
    // here knows how many.)
    const long long rows = (long long)max_q_len * (heads / kv_heads);
    if (dtype == MB_F32 && max_q_len > 1 && (head_dim == 64 || head_dim == 128) && q_row_stride % 4 == 0 && rows <= 0x7fffffff &&
        !(((uintptr_t)q | (uintptr_t)k_pool | (uintptr_t)v_pool) & 15))
        return (head_dim == 64 ? launch_row_tiles<64> : launch_row_tiles<128>)((const float*)q, q_row_stride, (float*)out, out_row_stride, (const float*)k_pool,
                                                                               (const float*)v_pool, block_table, max_blocks, cu_q, kv_lens, sequences, rows,
                                                                               heads, kv_heads, page_size, window, scale, stream);
    constexpr int kWarps = 4;
    const dim3 grid((max_q_len + kWarps - 1) / kWarps, heads, sequences);
    const size_t smem = (size_t)kWarps * head_dim * sizeof(float);
    if (dtype == MB_F32)
        paged_attention_rows_kernel<float, kWarps><<<grid, kWarps * 32, smem, stream>>>(
            (const float*)q, q_row_stride, (float*)out, out_row_stride, (const float*)k_pool, (const float*)v_pool,
            block_table, max_blocks, cu_q, kv_lens, heads, kv_heads, head_dim, page_size, window, scale);
    else if (dtype == MB_BF16)
        paged_attention_rows_kernel<__nv_bfloat16, kWarps><<<grid, kWarps * 32, smem, stream>>>(
            (const __nv_bfloat16*)q, q_row_stride, (__nv_bfloat16*)out, out_row_stride, (const __nv_bfloat16*)k_pool,
            (const __nv_bfloat16*)v_pool, block_table, max_blocks, cu_q, kv_lens, heads, kv_heads, head_dim, page_size,
            window, scale);
    else
        return fail("paged_attention_rows: unknown dtype code %d", dtype);
    return check_launch("paged_attention_rows");
}
