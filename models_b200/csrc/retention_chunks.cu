// Retention for long steps in bfloat16: chunks of 64 tokens on the tensor cores.  What is computed is what retention.cu's walk
// computes token by token (see there), for key heads of 64 numbers and value heads of 64 or 128:
//   S_t = a S_(t-1) + k_t v_t^T,   o_t = S_t^T q_t   (a: the head's decay; q, k, v activated, rotated and scaled as the walk does)
// and within a chunk that starts from the state S_0, for its token i = 0, 1, ...:
//   o_i = a^(i + 1) S_0^T q_i + sum_(j <= i) a^(i - j) (q_i . k_j) v_j,     S_end = a^n S_0 + sum_j a^(n - 1 - j) k_j v_j^T
// Three kernels: what every chunk adds to the state, a product per (chunk, head); the states that the chunks start from, element by
// element in the chunks' order; every chunk's results, with the head's norm and gate where the caller wants them here.
// The numbers between the first products and the last one are floats, and products take them whole (split_products.cuh).  A row that is
// not finite reaches its own and later tokens alone, as in the walk, where it may come out as NaN for an infinity.
// Against 64 bits, over steps of 64 to 2,048 tokens: the state is off by 6e-8 to 9e-8 of itself (the walk in runs: 0.9e-7 to 1.4e-7), the
// raw results by 0.7e-7 to 1.1e-7 (0.8e-7 to 1.8e-7); with two parts the operands would be cut to 16 bits.
// Three sequences of 2,048 tokens in all, 16 heads of 64 x 128 with activated projections: 208 us as the walk in runs (98, 70 and 40),
// which float multiply-adds from shared memory bound; here 24, 14 and 49 us (29, 14 and 54 with a division for every activation and a block's
// rows asked for one after the other), bound by the six products for one and by the instructions that activate and split what every chunk reads.
#include "common.cuh"
#include "gate_pairs.cuh"
#include "split_products.cuh"

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kChunk = 64;    // tokens of a chunk
constexpr int kDim = 64;      // a key head's numbers
constexpr int kThreads = 256;  // eight warps: four of 16 rows each for either half of the V columns
constexpr int kKeyRow = kDim + 8;                // bfloat16 numbers of a padded row: ldmatrix without bank conflicts
constexpr int kKeyPlane = kChunk * kKeyRow;      // one part of 64 rows; an operand's three planes lie one after another

template <int V>
struct Values {
    static constexpr int row = V + 8, plane = 64 * row;
};

struct RetentionArgs {
    const bf16 *q, *k, *v, *g;  // column slices with one row stride
    int in_stride;
    const int* positions;
    const float *cos_table, *sin_table;
    int rotary_dim;
    const float* decay;
    float key_scale, eps, out_scale;
    float* state;  // [slots][heads][kDim][V]
    const int *slots, *cu_q;
    int heads, input_act;
    bf16* out;
    int out_stride;
    float* raw_out;
    int raw_stride;
    float* starts;  // scratch by (place of the chunk, head): [kDim][V], what the chunk adds, then the state that it starts from
};

// Every sequence's chunks lie one after another, a sequence's first place being floor(first / 64) + seq (a sequence of n tokens has
// ceil(n / 64) chunks, and floor(f / 64) + ceil(n / 64) <= floor((f + n) / 64) + 1).
__device__ __forceinline__ size_t place_of(int first, int seq, int chunk) { return (size_t)(first / kChunk) + seq + chunk; }

// The queries or keys of `count` tokens (64 with zeros behind them) of a head, activated, rotated, times weight[row] (or 1), in planes.
__device__ __forceinline__ void stage_turned_rows(bf16* planes, const bf16* src, const RetentionArgs& args, int count, int position0, const float* weight) {
    const int rotary = args.rotary_dim, half = rotary / 2;
#pragma unroll 2
    for (int i = threadIdx.x; i < kChunk * kDim / 8; i += kThreads) {
        const int row = i / (kDim / 8), c = i % (kDim / 8) * 8;
        float x[8] = {0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f, 0.0f};
        if (row < count) {
            const bf16* from = src + (size_t)row * args.in_stride;
            load8(from + c, x);
            if (args.input_act >= 0)
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] = gate_activation(args.input_act, x[j]);
            if (c < rotary)
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    const int d = c + j;
                    if (d >= rotary) break;
                    const bool first = d < half;
                    float partner = __bfloat162float(from[first ? d + half : d - half]);
                    if (args.input_act >= 0) partner = gate_activation(args.input_act, partner);
                    const size_t at = (size_t)(position0 + row) * half + (first ? d : d - half);
                    x[j] = x[j] * args.cos_table[at] + (first ? -1.0f : 1.0f) * partner * args.sin_table[at];
                }
            const float factor = weight != nullptr ? weight[row] : 1.0f;
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] *= factor;
        }
        store_parts(planes + row * kKeyRow + c, kKeyPlane, x);
    }
}

// A thread's part of rows of kCols columns (values, and queries and keys without rotation): asked for, all of a block's rows before any is
// waited for, and later activated and put in place, the same numbers as above.
template <int kCols>
struct RawRows {
    static constexpr int kPieces = kChunk * kCols / 8 / kThreads;
    uint4 raw[kPieces];
    __device__ __forceinline__ void ask(const bf16* src, int stride, int count) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = threadIdx.x + i * kThreads, row = piece / (kCols / 8);
            raw[i] = make_uint4(0, 0, 0, 0);
            if (row < count) raw[i] = *reinterpret_cast<const uint4*>(src + (size_t)row * stride + piece % (kCols / 8) * 8);
        }
    }
    // Returns a sum that is finite only where every number is, and has three finite parts.  The pieces side by side, or (kOneByOne) by one body
    // of code: adds 23.0 -> 21.4 us so, but results of short steps 22.0 -> 24.2.
    template <bool kOneByOne>
    __device__ __forceinline__ float put(bf16* planes, int row_numbers, int plane_numbers, int activation, int count, const float* weight) {
        float fit = 0.0f;
#pragma unroll (kOneByOne ? 1 : kPieces)
        for (int i = 0; i < kPieces; ++i) {
            const int piece = threadIdx.x + i * kThreads, row = piece / (kCols / 8);
            const uint32_t w[4] = {raw[0].x, raw[0].y, raw[0].z, raw[0].w};
            move_up<1>(raw);
            float x[8];
#pragma unroll
            for (int j = 0; j < 4; ++j) x[2 * j] = __uint_as_float(w[j] << 16), x[2 * j + 1] = __uint_as_float(w[j] & 0xffff0000u);
            if (activation >= 0 && row < count) {
                const float ones[8] = {1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f, 1.0f};
                gate_pairs(activation, x, ones, ClampedPair{});
            }
            if (weight != nullptr)
#pragma unroll
                for (int j = 0; j < 8; ++j) x[j] *= weight[row];
            fit += fitness(x);
            store_parts(planes + row * row_numbers + piece % (kCols / 8) * 8, plane_numbers, x);
        }
        return fit;
    }
};

// grid (heads, most chunks of a sequence, sequences); block kThreads.  A warp has 16 coordinates and half of the columns of what the
// chunk adds.
template <int V>
__global__ void __launch_bounds__(kThreads)
retention_chunk_adds_kernel(const RetentionArgs args) {
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) unsigned char shared[];
    bf16* keys = reinterpret_cast<bf16*>(shared);
    bf16* values = keys + kParts * kKeyPlane;
    __shared__ float weight[kChunk];
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const bf16* key_rows = args.k + token0 * args.in_stride + (size_t)head * kDim;
    RawRows<V> v;
    RawRows<kDim> k;
    v.ask(args.v + token0 * args.in_stride + (size_t)head * V, args.in_stride, count);
    if (args.rotary_dim == 0) k.ask(key_rows, args.in_stride, count);
    if (tid < kChunk) weight[tid] = tid < count ? args.key_scale * powf(args.decay[head], (float)(count - 1 - tid)) : 0.0f;
    v.template put<true>(values, Values<V>::row, Values<V>::plane, args.input_act, count, nullptr);
    __syncthreads();
    if (args.rotary_dim == 0) k.template put<true>(keys, kKeyRow, kKeyPlane, args.input_act, count, weight);
    else stage_turned_rows(keys, key_rows, args, count, args.positions[first] + chunk * kChunk, weight);
    __syncthreads();
    const int tile = (tid >> 5) & 3, column0 = (tid >> 7) * (V / 2), lane = tid & 31;
    float acc[V / 16][4] = {};
    const uint32_t key_at = smem_u32(keys) + (((lane >> 4) * 8 + (lane & 7)) * kKeyRow + 16 * tile + ((lane >> 3) & 1) * 8) * 2;
    const uint32_t value_at = smem_u32(values) + ((lane & 15) * Values<V>::row + column0 + (lane >> 4) * 8) * 2;
#pragma unroll 1
    for (int j = 0; j < kChunk; j += 16) {
        Parts a, b;
        load_parts_turned(a, key_at + j * kKeyRow * 2, kKeyPlane);
#pragma unroll
        for (int n = 0; n < V / 16; n += 2) {
            load_parts_turned(b, value_at + (j * Values<V>::row + 8 * n) * 2, Values<V>::plane);
            split_products(acc[n], acc[n + 1], a, b);
        }
    }
    float* to = args.starts + (place_of(first, seq, chunk) * args.heads + head) * kDim * V + (size_t)(16 * tile + (lane >> 2)) * V + column0 + 2 * (lane & 3);
#pragma unroll
    for (int n = 0; n < V / 16; ++n) {
        *reinterpret_cast<float2*>(to + 8 * n) = make_float2(acc[n][0], acc[n][1]);
        *reinterpret_cast<float2*>(to + 8 * V + 8 * n) = make_float2(acc[n][2], acc[n][3]);
    }
}

// grid (kDim * V / 4 / 128, heads, sequences); block 128: four neighbouring elements a thread.  S before every chunk in the place of
// what the chunk adds, the state after the last one to the state area; eight chunks' additions are asked for at a time.
template <int V>
__global__ void __launch_bounds__(128)
retention_chunk_starts_kernel(const RetentionArgs args) {
    grid_launch_dependents();
    grid_dependency_wait();
    const int head = blockIdx.y, seq = blockIdx.z, e = (blockIdx.x * 128 + threadIdx.x) * 4;
    const int first = args.cu_q[seq], tokens = args.cu_q[seq + 1] - first;
    if (tokens <= 0) return;
    const int chunks = (tokens + kChunk - 1) / kChunk;
    const size_t item = place_of(first, seq, 0) * args.heads + head, stride = (size_t)args.heads * kDim * V;
    float* start = args.starts + item * kDim * V + e;
    float* stored = args.state + ((size_t)args.slots[seq] * args.heads + head) * kDim * V + e;
    const float a = args.decay[head], whole = powf(a, (float)kChunk), last = powf(a, (float)(tokens - (chunks - 1) * kChunk));
    float4 s = *reinterpret_cast<const float4*>(stored);
    constexpr int kAtOnce = 8;
    for (int c0 = 0; c0 < chunks; c0 += kAtOnce) {
        float4 b[kAtOnce];
#pragma unroll
        for (int i = 0; i < kAtOnce; ++i)
            if (c0 + i < chunks) b[i] = __ldcg(reinterpret_cast<const float4*>(start + (c0 + i) * stride));
#pragma unroll
        for (int i = 0; i < kAtOnce; ++i) {
            if (c0 + i >= chunks) break;
            *reinterpret_cast<float4*>(start + (c0 + i) * stride) = s;
            const float keep = c0 + i + 1 < chunks ? whole : last;
            s = make_float4(fmaf(keep, s.x, b[i].x), fmaf(keep, s.y, b[i].y), fmaf(keep, s.z, b[i].z), fmaf(keep, s.w, b[i].w));
        }
    }
    *reinterpret_cast<float4*>(stored) = s;
}

// grid (heads, most chunks of a sequence, sequences); block kThreads: a warp has 16 tokens and half of the V columns of their
// results (both halves' warps make the weights that they share).  The values take the start's place in shared memory, so that two blocks
// fit on a multiprocessor; they wait in registers until then.
template <int V>
__global__ void __launch_bounds__(kThreads, 2)
retention_chunk_results_kernel(const RetentionArgs args) {
    constexpr int kRow = Values<V>::row, kPlane = Values<V>::plane;
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) unsigned char shared[];
    bf16* queries = reinterpret_cast<bf16*>(shared);
    bf16* keys = queries + kParts * kKeyPlane;
    bf16* wide = keys + kParts * kKeyPlane;
    __shared__ float power[kChunk + 1], square_sums[2][kChunk];
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const bf16 *query_rows = args.q + token0 * args.in_stride + (size_t)head * kDim, *key_rows = args.k + token0 * args.in_stride + (size_t)head * kDim;
    RawRows<V> v;
    {
        constexpr int kPieces = 64 * V / 8 / kThreads;  // eights of the start that a thread brings
        const float* from = args.starts + (place_of(first, seq, chunk) * args.heads + head) * kDim * V;
        float x[kPieces][8];
        RawRows<kDim> q, k;
        if (args.rotary_dim == 0) q.ask(query_rows, args.in_stride, count), k.ask(key_rows, args.in_stride, count);
#pragma unroll
        for (int i = 0; i < kPieces; ++i) load8(from + 8 * (tid + i * kThreads), x[i]);
        v.ask(args.v + token0 * args.in_stride + (size_t)head * V, args.in_stride, count);
        if (tid <= kChunk) power[tid] = powf(args.decay[head], (float)tid);
        if (args.rotary_dim == 0) {
            q.template put<false>(queries, kKeyRow, kKeyPlane, args.input_act, count, nullptr);
            k.template put<false>(keys, kKeyRow, kKeyPlane, args.input_act, count, nullptr);
        } else {
            const int position0 = args.positions[first] + chunk * kChunk;
            stage_turned_rows(queries, query_rows, args, count, position0, nullptr);
            stage_turned_rows(keys, key_rows, args, count, position0, nullptr);
        }
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = tid + i * kThreads;
            store_parts(wide + piece / (V / 8) * kRow + piece % (V / 8) * 8, kPlane, x[i]);
        }
    }
    __syncthreads();
    const int warp = (tid >> 5) & 3, half_columns = tid >> 7, column0 = half_columns * (V / 2), lane = tid & 31, group = lane >> 2, pair = 2 * (lane & 3);
    const uint32_t query_at = smem_u32(queries) + ((16 * warp + (lane & 15)) * kKeyRow + (lane >> 4) * 8) * 2;
    const uint32_t wide_at = smem_u32(wide) + ((lane & 15) * kRow + column0 + (lane >> 4) * 8) * 2;  // [k][column] tiles of V columns
    const uint32_t key_at = smem_u32(keys) + (((lane >> 4) * 8 + (lane & 7)) * kKeyRow + ((lane >> 3) & 1) * 8) * 2;
    float acc[V / 16][4] = {}, weights[kChunk / 8][4] = {};
#pragma unroll 1
    for (int d = 0; d < kDim; d += 16) {
        Parts a, b;
        load_parts(a, query_at + d * 2, kKeyPlane);
#pragma unroll
        for (int n = 0; n < V / 16; n += 2) {  // S_0^T q
            load_parts_turned(b, wide_at + (d * kRow + 8 * n) * 2, kPlane);
            split_products(acc[n], acc[n + 1], a, b);
        }
#pragma unroll
        for (int n = 0; n < kChunk / 8; n += 2) {  // q . k over the tokens up to the warp's last
            if (n > 2 * warp) break;
            load_parts(b, key_at + (8 * n * kKeyRow + d) * 2, kKeyPlane);
            split_products(weights[n], weights[n + 1], a, b);
        }
    }
    __syncthreads();  // nobody reads the start any more
    const float fit = v.template put<false>(wide, kRow, kPlane, args.input_act, count, nullptr);
    const bool spoiled = __syncthreads_or(!isfinite(fit));
    const int row = 16 * warp + group;
#pragma unroll
    for (int n = 0; n < V / 16; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] *= power[row + 8 * (i / 2) + 1];
#pragma unroll 1
    for (int n = 0; n <= 2 * warp; n += 2) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int age = row + 8 * (i / 2) - (8 * (n + m) + pair + i % 2);
                weights[m][i] = age >= 0 ? weights[m][i] * (args.key_scale * power[max(age, 0)]) : 0.0f;
            }
        Parts a, b;
        split_pair(weights[0][0], weights[0][1], a[0][0], a[1][0], a[2][0]);
        split_pair(weights[0][2], weights[0][3], a[0][1], a[1][1], a[2][1]);
        split_pair(weights[1][0], weights[1][1], a[0][2], a[1][2], a[2][2]);
        split_pair(weights[1][2], weights[1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
        for (int c = 0; c < V / 16; c += 2) {
            load_parts_turned(b, wide_at + (8 * n * kRow + 8 * c) * 2, kPlane);
            split_products(acc[c], acc[c + 1], a, b);
        }
        move_up<2>(weights);
    }
    if (spoiled) {  // a value that is not finite: see causal_products
        auto weight = [&](int token, int from) {
            return whole_dot<kDim>(queries + token * kKeyRow, keys + from * kKeyRow, kKeyPlane) * (args.key_scale * power[token - from]);
        };
        start_products<kDim>(acc, queries + row * kKeyRow, kKeyRow, kKeyPlane,
                             args.starts + (place_of(first, seq, chunk) * args.heads + head) * kDim * V + column0 + pair, V);
#pragma unroll
        for (int n = 0; n < V / 16; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] *= power[row + 8 * (i / 2) + 1];
        causal_products(acc, row, weight, wide + column0 + pair, kRow, kPlane);
    }
    if (args.raw_out == nullptr) {  // a row's V results lie with four neighbouring lanes of two warps
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            float squares = 0.0f;
#pragma unroll
            for (int n = 0; n < V / 16; ++n) squares = fmaf(acc[n][2 * half], acc[n][2 * half], fmaf(acc[n][2 * half + 1], acc[n][2 * half + 1], squares));
            squares += __shfl_xor_sync(0xffffffffu, squares, 1);
            squares += __shfl_xor_sync(0xffffffffu, squares, 2);
            if (pair == 0) square_sums[half_columns][row + 8 * half] = squares;
        }
        __syncthreads();
    }
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int to = row + 8 * half;
        float factor = args.out_scale;
        if (args.raw_out == nullptr) factor /= sqrtf((square_sums[0][to] + square_sums[1][to]) / (float)V + args.eps);
        if (to >= count) continue;
        const size_t column = (size_t)head * V + column0 + pair;
        if (args.raw_out != nullptr) {
            float* dst = args.raw_out + (token0 + to) * args.raw_stride + column;
#pragma unroll
            for (int n = 0; n < V / 16; ++n) *reinterpret_cast<float2*>(dst + 8 * n) = make_float2(acc[n][2 * half] * factor, acc[n][2 * half + 1] * factor);
        } else {
            const bf16* gate = args.g + (token0 + to) * args.in_stride + column;
            bf16* dst = args.out + (token0 + to) * args.out_stride + column;
            uint32_t raw[V / 16];  // (all of them before the first store: one by one each waited for itself)
#pragma unroll
            for (int n = 0; n < V / 16; ++n) raw[n] = *reinterpret_cast<const uint32_t*>(gate + 8 * n);
#pragma unroll
            for (int n = 0; n < V / 16; n += 2) {
                float z[4] = {__uint_as_float(raw[n] << 16), __uint_as_float(raw[n] & 0xffff0000u), __uint_as_float(raw[n + 1] << 16), __uint_as_float(raw[n + 1] & 0xffff0000u)};
                const float ones[4] = {1.0f, 1.0f, 1.0f, 1.0f};
                gate_pairs(MB_ACT_SILU, z, ones, ClampedPair{});
#pragma unroll
                for (int m = n; m < n + 2; ++m)
                    *reinterpret_cast<__nv_bfloat162*>(dst + 8 * m) =
                        __floats2bfloat162_rn(acc[m][2 * half] * factor * z[2 * (m - n)], acc[m][2 * half + 1] * factor * z[2 * (m - n) + 1]);
            }
        }
    }
}

template <typename Kernel>
static int reserve(Kernel kernel, int bytes) {
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (status != cudaSuccess) return fail("retention_chunks: cannot reserve %d bytes of shared memory: %s", bytes, cudaGetErrorString(status));
    return 0;
}

template <int V>
static int launch_chunks(const RetentionArgs& args, int sequences, int chunks, cudaStream_t stream) {
    constexpr int adds = kParts * (kKeyPlane + Values<V>::plane) * 2, results = kParts * (2 * kKeyPlane + Values<V>::plane) * 2;
    if (int status = reserve(retention_chunk_adds_kernel<V>, adds)) return status;
    if (int status = reserve(retention_chunk_results_kernel<V>, results)) return status;
    const dim3 grid(args.heads, chunks, sequences);
    MB_LAUNCH("retention_chunks", (retention_chunk_adds_kernel<V>), grid, dim3(kThreads), adds, stream, true, args);
    MB_LAUNCH("retention_chunks", (retention_chunk_starts_kernel<V>), dim3(kDim * V / 512, args.heads, sequences), dim3(128), 0, stream, true, args);
    MB_LAUNCH("retention_chunks", (retention_chunk_results_kernel<V>), grid, dim3(kThreads), results, stream, true, args);
    return check_launch("retention_chunks");
}

}  // namespace mb

using namespace mb;

MB_EXPORT int mb_retention_chunk_tokens() { return kChunk; }

// Arguments as mb_retention_scan's, bfloat16 storage, head_dim 64, value_dim 64 or 128, whole aligned rows (see the checks).  starts:
// (places * heads * 64 * value_dim) floats, with places = tokens / 64 + sequences.
MB_EXPORT int mb_retention_chunks(const void* q, const void* k, const void* v, const void* g, int in_stride, const int* positions,
                                  const float* cos_table, const float* sin_table, int rotary_dim, const float* decay, float key_scale, float eps,
                                  float* state, const int* slots, const int* cu_q, int sequences, int heads, int head_dim, int value_dim, void* out,
                                  int out_stride, float out_scale, int max_q_len, float* starts, int input_act, float* raw_out,
                                  int raw_stride, cudaStream_t stream) {
    if (sequences <= 0 || heads <= 0 || max_q_len <= 0) return 0;
    if (input_act >= MB_ACT_COUNT) return fail("retention_chunks: unknown activation code %d", input_act);
    if (head_dim != kDim || (value_dim != 64 && value_dim != 128)) return fail("retention_chunks: heads of %d and %d numbers are not built (64 and 64 or 128 are)", head_dim, value_dim);
    if (rotary_dim < 0 || rotary_dim % 2 || rotary_dim > head_dim || (rotary_dim > 0 && (!cos_table || !sin_table)))
        return fail("retention_chunks: rotary_dim %d must be even, at most %d, and come with its tables", rotary_dim, head_dim);
    if (!raw_out && (!out || !g)) return fail("retention_chunks: results go to raw_out, or gated to out");
    const int chunks = (max_q_len + kChunk - 1) / kChunk;
    if (sequences > 65535 || chunks > 65535 || heads > 65535) return fail("retention_chunks: %d sequences of up to %d chunks and %d heads exceed the grid", sequences, chunks, heads);
    if (in_stride % 8 || ((uintptr_t)q & 15) || ((uintptr_t)k & 15) || ((uintptr_t)v & 15) || ((uintptr_t)state & 15) ||
        ((uintptr_t)starts & 15) || (raw_out && (raw_stride % 2 || ((uintptr_t)raw_out & 7))) ||
        (!raw_out && (out_stride % 2 || ((uintptr_t)out & 3) || ((uintptr_t)g & 3))))
        return fail("retention_chunks: rows of whole, aligned pieces are needed");
    RetentionArgs args{};
    args.q = (const bf16*)q, args.k = (const bf16*)k, args.v = (const bf16*)v, args.g = (const bf16*)g, args.in_stride = in_stride;
    args.positions = positions, args.cos_table = cos_table, args.sin_table = sin_table, args.rotary_dim = rotary_dim;
    args.decay = decay, args.key_scale = key_scale, args.eps = eps, args.out_scale = out_scale;
    args.state = state, args.slots = slots, args.cu_q = cu_q, args.heads = heads, args.input_act = input_act;
    args.out = (bf16*)out, args.out_stride = out_stride, args.raw_out = raw_out, args.raw_stride = raw_stride;
    args.starts = starts;
    return value_dim == 64 ? launch_chunks<64>(args, sequences, chunks, stream) : launch_chunks<128>(args, sequences, chunks, stream);
}
