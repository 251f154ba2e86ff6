// The gated delta rule for long steps: chunks of 64 tokens, float arithmetic throughout.  What is computed is what
// gated_delta.cu's walk computes token by token (see there):
//   S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
// Within a chunk that starts from the state S_0, with G_i the product of the chunk's g up to token i:
//   u_i = beta_i (v_i - G_i S_0^T k_i - sum_(j < i) G_i / G_j (k_i . k_j) u_j)
//   o_i = G_i S_0^T q_i + sum_(j <= i) G_i / G_j (q_i . k_j) u_j
//   S_end = G_end S_0 + sum_j G_end / G_j k_j u_j^T
// The first line is a triangular system in the chunk's u (the UT form of products of Householder-like factors: Bischof and
// Van Loan 1987; for delta rules Yang et al. 2024), linear in S_0: u = x - y S_0, where x and y solve it for the right sides
// beta v and beta G k.  Three kernels:
//   1. delta_chunks_solve: per (chunk, head) the system's matrix, x [64][V], y [64][64] and the keys weighted by G_end / G_j,
//      by forward substitution, a thread for every two columns of the right sides;
//   2. delta_chunks_carry: per (head, 16 columns of S) from chunk to chunk: u = x - y S_0 (over x), S_0 left for kernel 3,
//      S_end; the only serial part, two 64 x 64 x 16 products a chunk;
//   3. delta_chunks_results: per (chunk, head) o, its norm, gain and gate.
// The ratios G_i / G_j come from differences of sums of log g that are kept in 64 bits, so that a late token's ratios lose
// nothing to the size of the sums.
// One sequence of 2,048 tokens, 16 heads of 64 x 128: the walk's chain of 2,048 tokens is bound by its latency (618 us, and 30 for
// the kernels around it); here 56, 102 and 68 us, bound by what the operands take from shared memory (the carrying kernel: by the
// latency of two warps).
#include "common.cuh"

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kChunk = 64;    // tokens of a chunk
constexpr int kDim = 64;      // a key head's coordinates
constexpr int kColumns = 16;  // columns of S that a block of the carrying kernel owns
constexpr int kPad = 4;       // floats behind the rows of a transposed tile

struct DeltaChunkArgs {
    const float* conv;  // convolved rows: q at column q_at (kv_heads heads of kDim), k at k_at, v at v_at (heads heads of V)
    int conv_stride, q_at, k_at, v_at;
    const void *a_in, *b_in, *gate_in;
    int in_stride;
    const float *decay, *dt_bias, *gain;
    float unit_eps, eps, out_scale;
    float* state;
    size_t state_stride;
    const int *slots, *cu_q;
    void* out;
    int out_stride;
    int heads, kv_heads;
    // scratch, by (place of the chunk, head): u [64][V], y transposed [64 d][64 i], weighted keys [64 i][64 d], S_0 [64 d][V], sums of log g
    float *u, *y, *keys, *starts;
    double* logs;
};

__device__ __forceinline__ float sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus(float v) { return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v))); }

__device__ __forceinline__ uint64_t pair_of(float lo, float hi) {
    uint64_t d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(d) : "f"(lo), "f"(hi));
    return d;
}
__device__ __forceinline__ uint64_t twice(float v) { return pair_of(v, v); }
__device__ __forceinline__ float2 floats_of(uint64_t v) { return make_float2(__uint_as_float((uint32_t)v), __uint_as_float((uint32_t)(v >> 32))); }
__device__ __forceinline__ uint64_t fma_pair(uint64_t a, uint64_t b, uint64_t c) {  // two float FMAs
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ void copy16_async(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void copies_sent() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory");
}

// Where a chunk's scratch lies: every sequence's chunks one after another, a sequence's first place being floor(first / 64) + seq
// (a sequence of n tokens has ceil(n / 64) chunks, and floor(f / 64) + ceil(n / 64) <= floor((f + n) / 64) + 1).
__device__ __forceinline__ size_t place_of(int first, int seq, int chunk) { return (size_t)(first / kChunk) + seq + chunk; }

// The unit rows of a chunk's 64 tokens, times `factor`, transposed into tile [kDim][kChunk + kPad]; 128 threads, thread (row, half)
// takes 32 coordinates of a row and leaves them in `own` too.  Rows beyond `count` are zeros.  parts: shared [2][kChunk].
__device__ __forceinline__ void unit_rows(const float* rows, int stride, int count, float unit_eps, float factor, float* tile, float* parts,
                                          float (&own)[32]) {
    const int row = threadIdx.x % kChunk, half = threadIdx.x / kChunk;
    float squares = 0.0f;
#pragma unroll
    for (int i = 0; i < 32; i += 4) {
        const float4 x = row < count ? *reinterpret_cast<const float4*>(rows + (size_t)row * stride + half * 32 + i) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        own[i] = x.x, own[i + 1] = x.y, own[i + 2] = x.z, own[i + 3] = x.w;
        squares = fmaf(x.x, x.x, squares), squares = fmaf(x.y, x.y, squares), squares = fmaf(x.z, x.z, squares), squares = fmaf(x.w, x.w, squares);
    }
    parts[half * kChunk + row] = squares;
    __syncthreads();
    const float scale = factor / sqrtf(parts[row] + parts[kChunk + row] + unit_eps);
#pragma unroll
    for (int i = 0; i < 32; ++i) {
        own[i] *= scale;
        tile[(half * 32 + i) * (kChunk + kPad) + row] = own[i];
    }
}

// acc[8 rows][4 columns] += a^T b over 64 steps: a [64][kChunk + kPad] at rows row0 .. +3 and row0 + 32 .. +35, b likewise at col0 .. +3.
__device__ __forceinline__ void tile_8x4(const float* a, const float* b, int row0, int col0, uint64_t (&acc)[8][2]) {
#pragma unroll 8
    for (int d = 0; d < 64; ++d) {
        const float4 lo = *reinterpret_cast<const float4*>(a + d * (kChunk + kPad) + row0), hi = *reinterpret_cast<const float4*>(a + d * (kChunk + kPad) + row0 + 32);
        const ulonglong2 c = *reinterpret_cast<const ulonglong2*>(b + d * (kChunk + kPad) + col0);
        const float rows[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const uint64_t x = twice(rows[r]);
            acc[r][0] = fma_pair(x, c.x, acc[r][0]);
            acc[r][1] = fma_pair(x, c.y, acc[r][1]);
        }
    }
}

// grid (heads, most chunks of a sequence, sequences); block 128.
// shared: keys transposed [64][68], matrix transposed [j][i] [64][64], right sides [64][V + 64], sums of log g, beta, parts.
template <int V>
struct SolvePlan {
    static constexpr int kRight = V + kDim;
    static constexpr int keys = 0, matrix = keys + kDim * (kChunk + kPad), right = matrix + kChunk * kChunk, logs = right + kChunk * kRight,
                         beta = logs + 2 * kChunk, parts = beta + kChunk, total = parts + 2 * kChunk;
};

template <typename T, int V>
__global__ void __launch_bounds__(128)
delta_chunks_solve_kernel(const DeltaChunkArgs args) {
    using Plan = SolvePlan<V>;
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) float shared[];
    float* keys = shared + Plan::keys;
    float* matrix = shared + Plan::matrix;
    float* right = shared + Plan::right;
    double* logs = reinterpret_cast<double*>(shared + Plan::logs);
    float* beta = shared + Plan::beta;
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const size_t at = place_of(first, seq, chunk) * args.heads + head;
    const float* rows = args.conv + token0 * args.conv_stride;
    // gates: a token beyond the chunk's last neither forgets nor writes
    double log_g = 0.0;
    if (tid < kChunk) {
        float b = 0.0f;
        if (tid < count) {
            const size_t in = (token0 + tid) * args.in_stride + head;
            b = sigmoid(Num<T>::load((const T*)args.b_in + in));
            const float forget = args.decay[head] * softplus(Num<T>::load((const T*)args.a_in + in) + args.dt_bias[head]);
            log_g = (double)(forget < -1e6f ? -1e6f : forget);  // (g is zero long before; sums of infinities would have no difference)
        }
        beta[tid] = b;
        const int lane = tid & 31;
#pragma unroll
        for (int offset = 1; offset < 32; offset <<= 1) {
            const double other = __shfl_up_sync(0xffffffffu, log_g, offset);
            if (lane >= offset) log_g += other;
        }
        logs[tid] = log_g;
    }
    float own[32];
    unit_rows(rows + args.k_at + head / (args.heads / args.kv_heads) * kDim, args.conv_stride, count, args.unit_eps, 1.0f, keys, shared + Plan::parts, own);
    if (tid >= 32 && tid < kChunk) logs[tid] = log_g + logs[31];  // (the barrier inside unit_rows lies between)
    // the values' right sides: beta v
    for (int i = tid; i < kChunk * (V / 4); i += 128) {
        const int row = i / (V / 4), c = i % (V / 4) * 4;
        float4 v = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (row < count) v = *reinterpret_cast<const float4*>(rows + (size_t)row * args.conv_stride + args.v_at + (size_t)head * V + c);
        const float b = beta[row];
        *reinterpret_cast<float4*>(right + row * Plan::kRight + c) = make_float4(b * v.x, b * v.y, b * v.z, b * v.w);
    }
    __syncthreads();
    {
        // the keys' right sides beta G k, and the keys weighted for the chunk's end
        const int row = tid % kChunk, half = tid / kChunk;
        const float to_row = beta[row] * expf((float)logs[row]), to_end = expf((float)(logs[kChunk - 1] - logs[row]));
        float* weighted = args.keys + at * kChunk * kDim + row * kDim + half * 32;
#pragma unroll
        for (int i = 0; i < 32; i += 4) {
            *reinterpret_cast<float4*>(right + row * Plan::kRight + V + half * 32 + i) =
                make_float4(to_row * own[i], to_row * own[i + 1], to_row * own[i + 2], to_row * own[i + 3]);
            *reinterpret_cast<float4*>(weighted + i) = make_float4(to_end * own[i], to_end * own[i + 1], to_end * own[i + 2], to_end * own[i + 3]);
        }
        if (tid < kChunk) args.logs[at * kChunk + tid] = logs[tid];
    }
    {
        // matrix[j][i] = beta_i G_i / G_j (k_i . k_j) for j < i
        const int row0 = (tid % 8) * 4, col0 = (tid / 8) * 4;  // rows j, columns i
        uint64_t acc[8][2];
#pragma unroll
        for (int r = 0; r < 8; ++r) acc[r][0] = acc[r][1] = 0;
        tile_8x4(keys, keys, row0, col0, acc);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int j = row0 + (r / 4) * 32 + r % 4;
            const float2 lo = floats_of(acc[r][0]), hi = floats_of(acc[r][1]);
            float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
            for (int c = 0; c < 4; ++c) {
                const int i = col0 + c;
                v[c] = j < i ? v[c] * beta[i] * expf((float)(logs[i] - logs[j])) : 0.0f;
            }
            *reinterpret_cast<float4*>(matrix + j * kChunk + col0) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    __syncthreads();
    // forward substitution, 16 rows at a time; a thread's two columns are its own from here on
    for (int column = 2 * tid; column < Plan::kRight; column += 256) {
#pragma unroll 1
        for (int row0 = 0; row0 < kChunk; row0 += 16) {
            uint64_t acc[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) acc[r] = *reinterpret_cast<const uint64_t*>(right + (row0 + r) * Plan::kRight + column);
#pragma unroll 4
            for (int j = 0; j < row0; ++j) {
                const float2 x = *reinterpret_cast<const float2*>(right + j * Plan::kRight + column);
                const uint64_t minus = pair_of(-x.x, -x.y);
#pragma unroll
                for (int r = 0; r < 16; r += 4) {
                    const float4 m = *reinterpret_cast<const float4*>(matrix + j * kChunk + row0 + r);
                    acc[r] = fma_pair(twice(m.x), minus, acc[r]);
                    acc[r + 1] = fma_pair(twice(m.y), minus, acc[r + 1]);
                    acc[r + 2] = fma_pair(twice(m.z), minus, acc[r + 2]);
                    acc[r + 3] = fma_pair(twice(m.w), minus, acc[r + 3]);
                }
            }
#pragma unroll
            for (int j = 0; j < 16; ++j) {
                const float2 x = floats_of(acc[j]);
                const uint64_t minus = pair_of(-x.x, -x.y);
                *reinterpret_cast<uint64_t*>(right + (row0 + j) * Plan::kRight + column) = acc[j];
#pragma unroll
                for (int r = j + 1; r < 16; ++r) acc[r] = fma_pair(twice(matrix[(row0 + j) * kChunk + row0 + r]), minus, acc[r]);
            }
            if (column < V) {
#pragma unroll
                for (int r = 0; r < 16; ++r) *reinterpret_cast<uint64_t*>(args.u + (at * kChunk + row0 + r) * V + column) = acc[r];
            } else {
                float* y = args.y + at * kDim * kChunk + (size_t)(column - V) * kChunk + row0;  // transposed
#pragma unroll
                for (int r = 0; r < 16; r += 4) {
                    const float2 a = floats_of(acc[r]), b = floats_of(acc[r + 1]), c = floats_of(acc[r + 2]), d = floats_of(acc[r + 3]);
                    *reinterpret_cast<float4*>(y + r) = make_float4(a.x, b.x, c.x, d.x);
                    *reinterpret_cast<float4*>(y + kChunk + r) = make_float4(a.y, b.y, c.y, d.y);
                }
            }
        }
    }
}

// grid (V / kColumns, heads, sequences); block 64: thread (four, group) holds S at coordinates 4 * four .. +3 and columns
// 4 * group .. +3, and the same places of u.  The next chunk's y, keys and x arrive by cp.async while this one's are used.
template <int V>
__global__ void __launch_bounds__(64)
delta_chunks_carry_kernel(const DeltaChunkArgs args) {
    grid_launch_dependents();
    grid_dependency_wait();
    constexpr int kStage = 2 * kDim * kChunk + kChunk * kColumns;  // y, keys, x
    extern __shared__ __align__(16) float shared[];
    float* s_tile = shared + 2 * kStage;           // [64 d][16]
    float* u_tile = s_tile + kDim * kColumns;      // [64 i][16]
    const int column0 = blockIdx.x * kColumns, head = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], tokens = args.cu_q[seq + 1] - first;
    if (tokens <= 0) return;
    const int chunks = (tokens + kChunk - 1) / kChunk;
    const int four = (tid % 16) * 4, group = (tid / 16) * 4;
    const size_t place0 = place_of(first, seq, 0);
    float* stored = args.state + (size_t)args.slots[seq] * args.state_stride + (size_t)head * kDim * V + column0 + group;
    auto fetch = [&](int chunk) {
        float* stage = shared + (chunk & 1) * kStage;
        const size_t at = (place0 + chunk) * args.heads + head;
        const float *y = args.y + at * kDim * kChunk, *keys = args.keys + at * kChunk * kDim, *x = args.u + at * kChunk * V + column0;
#pragma unroll 8
        for (int i = tid; i < kDim * kChunk / 4; i += 64) {
            copy16_async(stage + 4 * i, y + 4 * i);
            copy16_async(stage + kDim * kChunk + 4 * i, keys + 4 * i);
        }
#pragma unroll
        for (int i = tid; i < kChunk * kColumns / 4; i += 64)
            copy16_async(stage + 2 * kDim * kChunk + 4 * i, x + (size_t)(i / (kColumns / 4)) * V + i % (kColumns / 4) * 4);
        copies_sent();
    };
    fetch(0);
    uint64_t s[4][2];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        const float* from = stored + (size_t)(four + r) * V;
        s[r][0] = pair_of(from[0], from[1]), s[r][1] = pair_of(from[2], from[3]);
    }
    for (int chunk = 0; chunk < chunks; ++chunk) {
        const size_t at = (place0 + chunk) * args.heads + head;
        float* start = args.starts + at * kDim * V + column0 + group;
#pragma unroll
        for (int r = 0; r < 4; ++r) {
            const ulonglong2 row = make_ulonglong2(s[r][0], s[r][1]);
            *reinterpret_cast<ulonglong2*>(s_tile + (four + r) * kColumns + group) = row;
            *reinterpret_cast<ulonglong2*>(start + (size_t)(four + r) * V) = row;
        }
        const float keep = expf((float)args.logs[at * kChunk + kChunk - 1]);
        if (chunk + 1 < chunks) {
            fetch(chunk + 1);  // (its buffer was last read before the barrier that closed the chunk before)
            copies_wait<1>();
        } else {
            copies_wait<0>();
        }
        __syncthreads();
        const float* stage = shared + (chunk & 1) * kStage;
        {
            uint64_t u[4][2];  // u = x - y S_0
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const ulonglong2 x = *reinterpret_cast<const ulonglong2*>(stage + 2 * kDim * kChunk + (four + r) * kColumns + group);
                u[r][0] = x.x, u[r][1] = x.y;
            }
#pragma unroll 16
            for (int d = 0; d < kDim; ++d) {
                const float4 y = *reinterpret_cast<const float4*>(stage + d * kChunk + four);
                const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(s_tile + d * kColumns + group);
                const float rows[4] = {y.x, y.y, y.z, y.w};
#pragma unroll
                for (int r = 0; r < 4; ++r) {
                    const uint64_t minus = twice(-rows[r]);
                    u[r][0] = fma_pair(minus, b.x, u[r][0]);
                    u[r][1] = fma_pair(minus, b.y, u[r][1]);
                }
            }
            float* to = args.u + at * kChunk * V + column0 + group;
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const ulonglong2 row = make_ulonglong2(u[r][0], u[r][1]);
                *reinterpret_cast<ulonglong2*>(u_tile + (four + r) * kColumns + group) = row;
                *reinterpret_cast<ulonglong2*>(to + (size_t)(four + r) * V) = row;
            }
        }
        __syncthreads();
        const uint64_t kept = twice(keep);
#pragma unroll
        for (int r = 0; r < 4; ++r) s[r][0] = fma_pair(kept, s[r][0], 0), s[r][1] = fma_pair(kept, s[r][1], 0);
#pragma unroll 16
        for (int i = 0; i < kChunk; ++i) {
            const float4 k = *reinterpret_cast<const float4*>(stage + kDim * kChunk + i * kDim + four);
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(u_tile + i * kColumns + group);
            const float rows[4] = {k.x, k.y, k.z, k.w};
#pragma unroll
            for (int r = 0; r < 4; ++r) {
                const uint64_t x = twice(rows[r]);
                s[r][0] = fma_pair(x, b.x, s[r][0]);
                s[r][1] = fma_pair(x, b.y, s[r][1]);
            }
        }
        __syncthreads();  // the chunk's buffers and tiles may be written again
    }
#pragma unroll
    for (int r = 0; r < 4; ++r) {
        float* to = stored + (size_t)(four + r) * V;
        const float2 lo = floats_of(s[r][0]), hi = floats_of(s[r][1]);
        to[0] = lo.x, to[1] = lo.y, to[2] = hi.x, to[3] = hi.y;
    }
}

template <typename T>
__device__ __forceinline__ float4 load4(const T* p);
template <>
__device__ __forceinline__ float4 load4<float>(const float* p) { return *reinterpret_cast<const float4*>(p); }
template <>
__device__ __forceinline__ float4 load4<__nv_bfloat16>(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u), __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
}
__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    const __nv_bfloat162 a = __floats2bfloat162_rn(v.x, v.y), b = __floats2bfloat162_rn(v.z, v.w);
    *reinterpret_cast<uint2*>(p) = make_uint2(*reinterpret_cast<const uint32_t*>(&a), *reinterpret_cast<const uint32_t*>(&b));
}

// grid (heads, most chunks of a sequence, sequences); block 128: thread (rows 4 * (tid / 16) .. +3 and 32 on, columns
// 4 * (tid % 16) .. +3 of every 64).  shared: queries and keys transposed [64][68] (the second becomes the products' weights
// [j][i]), one [64][V] tile for S_0 and then u, sums of log g, parts.
template <int V>
struct ResultPlan {
    static constexpr int queries = 0, keys = queries + kDim * (kChunk + kPad), tile = keys + kDim * (kChunk + kPad), logs = tile + kDim * V,
                         parts = logs + 2 * kChunk, total = parts + 2 * kChunk;
};

template <typename T, int V>
__global__ void __launch_bounds__(128)
delta_chunks_results_kernel(const DeltaChunkArgs args) {
    using Plan = ResultPlan<V>;
    constexpr int kFours = V / 64;
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) float shared[];
    float* queries = shared + Plan::queries;
    float* keys = shared + Plan::keys;
    float* tile = shared + Plan::tile;
    double* logs = reinterpret_cast<double*>(shared + Plan::logs);
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const size_t at = place_of(first, seq, chunk) * args.heads + head;
    auto bring = [&](const float* from) {
#pragma unroll 8
        for (int i = tid; i < 64 * V / 4; i += 128) copy16_async(tile + 4 * i, from + 4 * i);
        copies_sent();
    };
    bring(args.starts + at * kDim * V);
    if (tid < kChunk) logs[tid] = args.logs[at * kChunk + tid];
    const float* rows = args.conv + token0 * args.conv_stride;
    const int qk_head = head / (args.heads / args.kv_heads);
    {
        float own[32];
        unit_rows(rows + args.k_at + qk_head * kDim, args.conv_stride, count, args.unit_eps, 1.0f, keys, shared + Plan::parts, own);
        __syncthreads();
        unit_rows(rows + args.q_at + qk_head * kDim, args.conv_stride, count, args.unit_eps, 0.125f, queries, shared + Plan::parts, own);  // 64^(-1/2)
    }
    copies_wait<0>();
    __syncthreads();
    const int row0 = (tid / 16) * 4, col0 = (tid % 16) * 4;
    uint64_t acc[8][2 * kFours];
#pragma unroll
    for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int c = 0; c < 2 * kFours; ++c) acc[r][c] = 0;
    auto product = [&](const float* a) {  // acc += a^T tile
#pragma unroll 4
        for (int d = 0; d < 64; ++d) {
            const float4 lo = *reinterpret_cast<const float4*>(a + d * (kChunk + kPad) + row0), hi = *reinterpret_cast<const float4*>(a + d * (kChunk + kPad) + row0 + 32);
            const float left[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            ulonglong2 b[kFours];
#pragma unroll
            for (int f = 0; f < kFours; ++f) b[f] = *reinterpret_cast<const ulonglong2*>(tile + d * V + 64 * f + col0);
#pragma unroll
            for (int r = 0; r < 8; ++r) {
                const uint64_t x = twice(left[r]);
#pragma unroll
                for (int f = 0; f < kFours; ++f) {
                    acc[r][2 * f] = fma_pair(x, b[f].x, acc[r][2 * f]);
                    acc[r][2 * f + 1] = fma_pair(x, b[f].y, acc[r][2 * f + 1]);
                }
            }
        }
    };
    product(queries);  // S_0^T q
    __syncthreads();   // the tile may be written again
    bring(args.u + at * kChunk * V);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const uint64_t g = twice(expf((float)logs[row0 + (r / 4) * 32 + r % 4]));
#pragma unroll
        for (int c = 0; c < 2 * kFours; ++c) acc[r][c] = fma_pair(g, acc[r][c], 0);
    }
    {
        // weights[j][i] = G_i / G_j (q_i . k_j) for j <= i, over the keys
        const int j0 = (tid % 8) * 4, i0 = (tid / 8) * 4;
        uint64_t w[8][2];
#pragma unroll
        for (int r = 0; r < 8; ++r) w[r][0] = w[r][1] = 0;
        tile_8x4(keys, queries, j0, i0, w);
        __syncthreads();  // everybody has read the keys
#pragma unroll
        for (int r = 0; r < 8; ++r) {
            const int j = j0 + (r / 4) * 32 + r % 4;
            const float2 lo = floats_of(w[r][0]), hi = floats_of(w[r][1]);
            float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
            for (int c = 0; c < 4; ++c) v[c] = j <= i0 + c ? v[c] * expf((float)(logs[i0 + c] - logs[j])) : 0.0f;
            *reinterpret_cast<float4*>(keys + j * (kChunk + kPad) + i0) = make_float4(v[0], v[1], v[2], v[3]);
        }
    }
    copies_wait<0>();
    __syncthreads();
    product(keys);
    // a row's V results lie with sixteen neighbouring lanes
    const T* gate = (const T*)args.gate_in + token0 * args.in_stride + (size_t)head * V;
    T* out = (T*)args.out + token0 * args.out_stride + (size_t)head * V;
#pragma unroll
    for (int r = 0; r < 8; ++r) {
        const int row = row0 + (r / 4) * 32 + r % 4;
        float squares = 0.0f;
#pragma unroll
        for (int c = 0; c < 2 * kFours; ++c) {
            const float2 o = floats_of(acc[r][c]);
            squares = fmaf(o.x, o.x, squares), squares = fmaf(o.y, o.y, squares);
        }
#pragma unroll
        for (int offset = 1; offset < 16; offset <<= 1) squares += __shfl_xor_sync(0xffffffffu, squares, offset);
        if (row < count) {
            const float inv = args.out_scale / sqrtf(squares / (float)V + args.eps);
#pragma unroll
            for (int f = 0; f < kFours; ++f) {
                const int c = 64 * f + col0;
                const float4 z = load4<T>(gate + (size_t)row * args.in_stride + c), gain = *reinterpret_cast<const float4*>(args.gain + c);
                const float2 lo = floats_of(acc[r][2 * f]), hi = floats_of(acc[r][2 * f + 1]);
                store4(out + (size_t)row * args.out_stride + c,
                       make_float4(lo.x * inv * gain.x * (z.x * sigmoid(z.x)), lo.y * inv * gain.y * (z.y * sigmoid(z.y)),
                                   hi.x * inv * gain.z * (z.z * sigmoid(z.z)), hi.y * inv * gain.w * (z.w * sigmoid(z.w))));
            }
        }
    }
}

template <typename Kernel>
static int reserve(Kernel kernel, int bytes) {
    cudaError_t status = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
    if (status != cudaSuccess) return fail("gated_delta_chunks: cannot reserve %d bytes of shared memory: %s", bytes, cudaGetErrorString(status));
    return 0;
}

template <typename T, int V>
static int launch_chunks(const DeltaChunkArgs& args, int sequences, int chunks, cudaStream_t stream) {
    constexpr int solve = SolvePlan<V>::total * 4, carry = (2 * (2 * kDim * kChunk + kChunk * kColumns) + (kDim + kChunk) * kColumns) * 4,
                  results = ResultPlan<V>::total * 4;
    if (int status = reserve(delta_chunks_solve_kernel<T, V>, solve)) return status;
    if (int status = reserve(delta_chunks_carry_kernel<V>, carry)) return status;
    if (int status = reserve(delta_chunks_results_kernel<T, V>, results)) return status;
    const dim3 grid(args.heads, chunks, sequences);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_solve_kernel<T, V>), grid, dim3(128), solve, stream, true, args);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_carry_kernel<V>), dim3(V / kColumns, args.heads, sequences), dim3(64), carry, stream, true, args);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_results_kernel<T, V>), grid, dim3(128), results, stream, true, args);
    return check_launch("gated_delta_chunks");
}

}  // namespace mb

using namespace mb;

MB_EXPORT int mb_gated_delta_chunk_tokens() { return kChunk; }

// Arguments as mb_gated_delta_scan's, with key heads of 64 numbers and value heads of 64 or 128; conv is only read.  scratch: floats,
// (places * heads) * (2 * 64 * vdim + 2 * 64 * 64 + 128), 16-byte aligned, with places = tokens / 64 + sequences.
MB_EXPORT int mb_gated_delta_chunks(const float* conv, int conv_stride, const void* a_in, const void* b_in, const void* gate_in, int in_stride,
                                    int dtype, const float* decay, const float* dt_bias, const float* gain, float unit_eps, float eps, float* state,
                                    size_t state_stride, const int* slots, const int* cu_q, int sequences, int tokens, int max_q_len, float* scratch,
                                    void* out, int out_stride, float out_scale, int heads, int kv_heads, int dim, int vdim, int q_at, int k_at,
                                    int v_at, cudaStream_t stream) {
    if (sequences <= 0 || heads <= 0 || tokens <= 0 || max_q_len <= 0) return 0;
    if (kv_heads <= 0 || heads % kv_heads) return fail("gated_delta_chunks: %d heads are no multiple of %d query/key heads", heads, kv_heads);
    if (dim != kDim || (vdim != 64 && vdim != 128)) return fail("gated_delta_chunks: heads of %d and %d numbers are not built (64 and 64 or 128 are)", dim, vdim);
    const int chunks = (max_q_len + kChunk - 1) / kChunk;
    if (sequences > 65535 || chunks > 65535 || heads > 65535) return fail("gated_delta_chunks: %d sequences of up to %d chunks and %d heads exceed the grid", sequences, chunks, heads);
    const size_t element = dtype == MB_F32 ? 4 : 2;
    if (conv_stride % 4 || q_at % 4 || k_at % 4 || v_at % 4 || in_stride % 4 || out_stride % 4 || ((uintptr_t)conv & 15) || ((uintptr_t)scratch & 15) ||
        ((uintptr_t)gain & 15) || (uintptr_t)gate_in % (4 * element) || (uintptr_t)out % (4 * element))
        return fail("gated_delta_chunks: rows of whole, aligned fours are needed");
    DeltaChunkArgs args{};
    args.conv = conv, args.conv_stride = conv_stride, args.q_at = q_at, args.k_at = k_at, args.v_at = v_at;
    args.a_in = a_in, args.b_in = b_in, args.gate_in = gate_in, args.in_stride = in_stride;
    args.decay = decay, args.dt_bias = dt_bias, args.gain = gain, args.unit_eps = unit_eps, args.eps = eps, args.out_scale = out_scale;
    args.state = state, args.state_stride = state_stride, args.slots = slots, args.cu_q = cu_q;
    args.out = out, args.out_stride = out_stride, args.heads = heads, args.kv_heads = kv_heads;
    const size_t items = ((size_t)tokens / kChunk + sequences) * heads;
    args.u = scratch;
    args.starts = args.u + items * kChunk * vdim;
    args.y = args.starts + items * kDim * vdim;
    args.keys = args.y + items * kDim * kChunk;
    args.logs = reinterpret_cast<double*>(args.keys + items * kChunk * kDim);
    if (dtype == MB_F32) return vdim == 64 ? launch_chunks<float, 64>(args, sequences, chunks, stream) : launch_chunks<float, 128>(args, sequences, chunks, stream);
    if (dtype == MB_BF16)
        return vdim == 64 ? launch_chunks<__nv_bfloat16, 64>(args, sequences, chunks, stream) : launch_chunks<__nv_bfloat16, 128>(args, sequences, chunks, stream);
    return fail("gated_delta_chunks: unknown dtype code %d", dtype);
}
