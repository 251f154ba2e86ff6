// The gated delta rule for long steps: chunks of 64 tokens on the tensor cores.  What is computed is what
// gated_delta.cu's walk computes token by token (see there):
//   S <- g_t S;   u_t = beta_t (v_t - S^T k_t);   S <- S + k_t u_t^T;   o_t = S^T q_t
// Within a chunk that starts from the state S_0, with G_i the product of the chunk's g up to token i:
//   u_i = beta_i (v_i - G_i S_0^T k_i - sum_(j < i) G_i / G_j (k_i . k_j) u_j)
//   o_i = G_i S_0^T q_i + sum_(j <= i) G_i / G_j (q_i . k_j) u_j
//   S_end = G_end S_0 + sum_j G_end / G_j k_j u_j^T
// The first line is a triangular system in the chunk's u (the UT form of products of Householder-like factors: Bischof and
// Van Loan 1987; for delta rules Yang et al. 2024), linear in S_0: u = x - y S_0, where x and y solve it for the right sides
// beta v and beta G k.  Three kernels:
//   1. delta_chunks_solve: per (chunk, head) the system's matrix, x [64][V], y [64][64] and the keys weighted by G_end / G_j; the
//      system is solved 16 rows at a time, with the inverses of its 16 x 16 diagonal blocks, a warp for 32 of the right sides'
//      columns;
//   2. delta_chunks_carry: per (head, 16 columns of S) from chunk to chunk: u = x - y S_0 (over x), S_0 left for kernel 3, S_end; the
//      only serial part, two 64 x 64 x 16 products a chunk;
//   3. delta_chunks_results: per (chunk, head) o, its norm, gain and gate.
// The ratios G_i / G_j come from differences of sums of log g that are kept in 64 bits, so that a late token's ratios lose
// nothing to the size of the sums.  What lies between products is float, and products take it whole (split_products.cuh).  A row that is
// not finite reaches its own and later tokens alone, as in the walk, where it may come out as NaN for an infinity.
// Against 64 bits, over steps of 64 to 2,048 tokens: the state is off by 1.2e-7 to 1.3e-7 of itself (the walk: 1.9e-7 to 3.3e-7), the
// results by 1.4e-7 (2e-7).
// One sequence of 2,048 tokens, 16 heads of 64 x 128: the walk's chain of 2,048 tokens is bound by its latency (618 us, and 30 for
// the kernels around it); the three kernels took 58, 105 and 71 us as float multiply-adds, bound by what the operands take from
// shared memory and by the latency of few warps; 37, 46 and 52 here (a layer: 310 us, and 199; 47, 46 and 58 and 221 with every loop unrolled
// and a block's gates asked for one by one), where the carrying kernel is bound by its chunk's two products one after the other, the others
// by six products for one and by the latency of what each phase of a block waits for.
#include "common.cuh"
#include "gate_pairs.cuh"
#include "split_products.cuh"

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kChunk = 64;    // tokens of a chunk
constexpr int kDim = 64;      // a key head's coordinates
constexpr int kColumns = 16;  // columns of S that a block of the carrying kernel owns
constexpr int kCarryThreads = 256, kResultThreads = 256;
constexpr int kRow = kDim + 8;            // bfloat16 numbers of a padded row of 64: ldmatrix without bank conflicts
constexpr int kPlane = kChunk * kRow;
constexpr int kNarrowRow = kColumns + 8;  // and of rows of 16
constexpr int kNarrowPlane = kChunk * kNarrowRow;

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
    // scratch by (place of the chunk, head): x, then u [64][V]; S_0 [64][V]; in three parts y [64 i][64 d] and weighted keys [64 i][64 d], as
    // `turned` says; sums of log g [64]
    float *u, *starts;
    bf16 *y, *keys;
    double* logs;
};

__device__ __forceinline__ float sigmoid(float v) { return 1.0f / (1.0f + expf(-v)); }
__device__ __forceinline__ float softplus(float v) { return fmaxf(v, 0.0f) + log1pf(expf(-fabsf(v))); }

template <typename T>
struct Pairs;  // two numbers as they are stored
template <>
struct Pairs<float> {
    using type = float2;
};
template <>
struct Pairs<bf16> {
    using type = uint32_t;
};
template <typename T>
using Pair = typename Pairs<T>::type;
__device__ __forceinline__ float2 load_pair(const float* p) { return *reinterpret_cast<const float2*>(p); }
__device__ __forceinline__ float2 load_pair(const bf16* p) { return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(p)); }
__device__ __forceinline__ void store_pair(float* p, float a, float b) { *reinterpret_cast<float2*>(p) = make_float2(a, b); }
__device__ __forceinline__ void store_pair(bf16* p, float a, float b) { *reinterpret_cast<__nv_bfloat162*>(p) = __floats2bfloat162_rn(a, b); }

// Where a chunk's scratch lies: every sequence's chunks one after another, a sequence's first place being floor(first / 64) + seq
// (a sequence of n tokens has ceil(n / 64) chunks, and floor(f / 64) + ceil(n / 64) <= floor((f + n) / 64) + 1).
__device__ __forceinline__ size_t place_of(int first, int seq, int chunk) { return (size_t)(first / kChunk) + seq + chunk; }

// Where number d of row i of a plane of y or of keys lies: the carrying kernel copies planes as they are, and its ldmatrix reads rows of 128
// bytes without bank conflicts if their 16-byte units are turned by the row.
__device__ __forceinline__ int turned(int i, int d) { return i * kDim + ((d >> 3 ^ (i & 7)) << 3) + (d & 7); }

// Four floats as their parts.
__device__ __forceinline__ void split_four(float4 v, bf16* at, int plane) {
    uint2 hi, mid, lo;
    split_pair(v.x, v.y, hi.x, mid.x, lo.x);
    split_pair(v.z, v.w, hi.y, mid.y, lo.y);
    *reinterpret_cast<uint2*>(at) = hi;
    *reinterpret_cast<uint2*>(at + plane) = mid;
    *reinterpret_cast<uint2*>(at + 2 * plane) = lo;
}

// The unit rows of a chunk's 64 tokens, times `factor`, into planes of padded rows; sixteen lanes a row, a thread's four coordinates of
// every row that it takes are left in `x`.  Rows beyond `count` are zeros.  unit (or null): the rows' factors.
template <int kThreads>
struct UnitRows {
    static constexpr int at_once = kThreads / 16, passes = (kChunk + at_once - 1) / at_once;
    float4 x[passes];
    __device__ __forceinline__ UnitRows(const float* rows, int stride, int count) {  // asks for the rows
        const int d = (threadIdx.x % 16) * 4;
#pragma unroll
        for (int i = 0; i < passes; ++i) {
            const int row = threadIdx.x / 16 + at_once * i;
            x[i] = row < count ? *reinterpret_cast<const float4*>(rows + (size_t)row * stride + d) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void put(int count, float unit_eps, float factor, bf16* planes, float* unit) {
        const int d = (threadIdx.x % 16) * 4;
#pragma unroll
        for (int i = 0; i < passes; ++i) {
            const int row = threadIdx.x / 16 + at_once * i;
            float squares = fmaf(x[i].x, x[i].x, fmaf(x[i].y, x[i].y, fmaf(x[i].z, x[i].z, x[i].w * x[i].w)));
#pragma unroll
            for (int offset = 1; offset < 16; offset <<= 1) squares += __shfl_xor_sync(0xffffffffu, squares, offset);
            const float scale = row < count ? factor / sqrtf(squares + unit_eps) : 0.0f;  // (unit_eps may be zero)
            x[i] = make_float4(scale * x[i].x, scale * x[i].y, scale * x[i].z, scale * x[i].w);
            if (row >= kChunk) continue;
            split_four(x[i], planes + row * kRow + d, kPlane);
            if (unit != nullptr && d == 0) unit[row] = scale;
        }
    }
};

// Where a lane's ldmatrix addresses start within a tile of rows of `row` numbers, in bytes: of a left operand [row][k] or a right one
// [k][column], and of a right one [column][k] or a left one [k][row].
__device__ __forceinline__ uint32_t lanes_by_row(int row) { return (((threadIdx.x & 31) & 15) * row + ((threadIdx.x & 31) >> 4) * 8) * 2; }
__device__ __forceinline__ uint32_t lanes_by_column(int row) {
    const int lane = threadIdx.x & 31;
    return (((lane >> 4) * 8 + (lane & 7)) * row + ((lane >> 3) & 1) * 8) * 2;
}

// grid (heads, most chunks of a sequence, sequences); block threads: a warp for 32 columns of the right sides.
template <int V>
struct SolvePlan {
    static constexpr int right = V + kDim, threads = right, right_row = right + 8, solved_rows = 48, right_plane = solved_rows * right_row;
    static constexpr int inverse_row = 24, inverse_plane = kChunk * inverse_row, diagonal_row = 17;
    // bfloat16 numbers: the matrix, the inverses of its diagonal blocks; the keys, whose place the solved rows take; then floats: the
    // diagonal blocks, beta, the keys' factors, (64 bits) logs
    static constexpr int matrix = 0, inverse = matrix + kParts * kPlane, keys = inverse + kParts * inverse_plane,
                         floats = keys + kParts * (right_plane > kPlane ? right_plane : kPlane);
    static constexpr int bytes = floats * 2 + (kChunk * diagonal_row + 2 * kChunk) * 4 + kChunk * 8;
    static_assert(floats * 2 % 16 == 0 && (kChunk * diagonal_row + 2 * kChunk) % 2 == 0, "the logs lie on eight bytes");
};

template <typename T, int V>
__global__ void __launch_bounds__(SolvePlan<V>::threads, 2)
delta_chunks_solve_kernel(const DeltaChunkArgs args) {
    using Plan = SolvePlan<V>;
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) unsigned char shared[];
    bf16* planes = reinterpret_cast<bf16*>(shared);
    bf16 *keys = planes + Plan::keys, *matrix = planes + Plan::matrix, *inverse = planes + Plan::inverse, *solved = keys;
    float* diagonal = reinterpret_cast<float*>(planes + Plan::floats);
    float* beta = diagonal + kChunk * Plan::diagonal_row;
    float* unit = beta + kChunk;
    double* logs = reinterpret_cast<double*>(unit + kChunk);
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const size_t at = place_of(first, seq, chunk) * args.heads + head;
    const float* rows = args.conv + token0 * args.conv_stride;
    const float* key_rows = rows + args.k_at + head / (args.heads / args.kv_heads) * kDim;
    const float* value_rows = rows + args.v_at + (size_t)head * V;
    UnitRows<Plan::threads> k(key_rows, args.conv_stride, count);
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
    k.put(count, args.unit_eps, 1.0f, keys, unit);
    __syncthreads();
    if (tid >= 32 && tid < kChunk) logs[tid] = log_g + logs[31];
    __syncthreads();
    {
        bf16* weighted = args.keys + kParts * at * kChunk * kDim;
#pragma unroll
        for (int i = 0; i < k.passes; ++i) {
            const int row = tid / 16 + k.at_once * i;
            if (row >= kChunk) break;
            const float to_end = expf((float)(logs[kChunk - 1] - logs[row]));
            split_four(make_float4(to_end * k.x[i].x, to_end * k.x[i].y, to_end * k.x[i].z, to_end * k.x[i].w), weighted + turned(row, (tid % 16) * 4), kChunk * kDim);
        }
        if (tid < kChunk) args.logs[at * kChunk + tid] = logs[tid];
    }
    const int warp = tid >> 5, group = (tid & 31) >> 2, pair = 2 * (tid & 3);
    // matrix[i][j] = beta_i G_i / G_j (k_i . k_j) for j < i: of every 16 rows the columns up to them, 16 a warp at a time
    for (int unit_at = warp; unit_at < 10; unit_at += Plan::threads / 32) {
        const int rows16 = unit_at >= 6 ? 3 : unit_at >= 3 ? 2 : unit_at >= 1 ? 1 : 0, columns16 = unit_at - rows16 * (rows16 + 1) / 2;
        float acc[2][4] = {};
        const uint32_t left = smem_u32(keys) + 16 * rows16 * kRow * 2 + lanes_by_row(kRow), right = smem_u32(keys) + 16 * columns16 * kRow * 2 + lanes_by_column(kRow);
#pragma unroll 1
        for (int d = 0; d < kDim; d += 16) {
            Parts a, b;
            load_parts(a, left + d * 2, kPlane);
            load_parts(b, right + d * 2, kPlane);
            split_products(acc[0], acc[1], a, b);
        }
#pragma unroll
        for (int n = 0; n < 2; ++n)
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int i = 16 * rows16 + group + 8 * half, j = 16 * columns16 + 8 * n + pair;
                const float b = beta[i];
                const float lo = j < i ? acc[n][2 * half] * b * expf((float)(logs[i] - logs[j])) : 0.0f;
                const float hi = j + 1 < i ? acc[n][2 * half + 1] * b * expf((float)(logs[i] - logs[j + 1])) : 0.0f;
                split_two(lo, hi, matrix + i * kRow + j, kPlane);
                if (columns16 == rows16) diagonal[i * Plan::diagonal_row + j % 16] = lo, diagonal[i * Plan::diagonal_row + j % 16 + 1] = hi;
            }
    }
    // a warp's columns of the right sides, beta v and beta G k, as products leave their results; all four blocks of 16 rows
    constexpr int kTiles = 4;  // tiles of eight columns
    const int column0 = warp * kTiles * 8;
    const bool of_values = column0 < V;
    const float* source = of_values ? value_rows + column0 + pair : key_rows + column0 - V + pair;
    float right[kChunk / 16][kTiles][4];
#pragma unroll
    for (int r = 0; r < kChunk / 8; ++r) {
        const int row = 8 * r + group;
#pragma unroll
        for (int n = 0; n < kTiles; ++n) {
            float2 x = make_float2(0.0f, 0.0f);
            if (row < count) x = load_pair(source + (size_t)row * args.conv_stride + 8 * n);
            const float scale = of_values ? beta[row] : beta[row] * expf((float)logs[row]) * unit[row];
            right[r / 2][n][2 * (r % 2)] = scale * x.x, right[r / 2][n][2 * (r % 2) + 1] = scale * x.y;
        }
    }
    __syncthreads();
    if (tid < kChunk) {
        // a column of the inverse of a diagonal block I + M: z_r = (r == c) - sum_(s < r) M[r][s] z_s
        const int block = tid / 16, c = tid % 16;
        float z[16] = {};
#pragma unroll 1
        for (int r = 0; r < 16; ++r) {
            float sum = r == c ? 1.0f : 0.0f;
#pragma unroll
            for (int s = 0; s < 16; ++s) sum = fmaf(-diagonal[(16 * block + r) * Plan::diagonal_row + s], z[s], sum);  // (from s = r on zeros meet zeros)
#pragma unroll
            for (int s = 0; s < 16; ++s) z[s] = s == r ? sum : z[s];
            uint32_t hi, mid, lo;
            split_pair(sum, 0.0f, hi, mid, lo);
            unsigned short* to = reinterpret_cast<unsigned short*>(inverse + (16 * block + r) * Plan::inverse_row + c);
            to[0] = (unsigned short)hi, to[Plan::inverse_plane] = (unsigned short)mid, to[2 * Plan::inverse_plane] = (unsigned short)lo;
        }
    }
    __syncthreads();  // (nobody reads the keys any more either)
    // a warp's columns are its own from here on; a block of 16 rows: z = right - sum over the blocks before of M x, x = inverse . z.  The
    // last block's z takes the first one's place, which nothing reads after it.
    const uint32_t matrix_at = smem_u32(matrix) + lanes_by_row(kRow), inverse_at = smem_u32(inverse) + lanes_by_row(Plan::inverse_row),
                   solved_at = smem_u32(solved) + column0 * 2 + lanes_by_row(Plan::right_row);
    float fit = 0.0f;
    // (Rolled loops: see move_up.)
#pragma unroll 1
    for (int block = 0; block < kChunk / 16; ++block) {
        const int row0 = 16 * block < Plan::solved_rows ? 16 * block : 0;
        float acc[kTiles][4] = {};
        auto accumulate = [&](uint32_t left, int left_plane, int k0) {  // acc += left (16 x 16) . rows k0 .. k0 + 15 of the solved columns
            Parts a, b;
            load_parts(a, left, left_plane);
#pragma unroll
            for (int n = 0; n < kTiles; n += 2) {
                load_parts_turned(b, solved_at + (k0 * Plan::right_row + 8 * n) * 2, Plan::right_plane);
                split_products(acc[n], acc[n + 1], a, b);
            }
        };
#pragma unroll 1
        for (int c = 0; c < block; ++c) accumulate(matrix_at + (16 * block * kRow + 16 * c) * 2, kPlane, 16 * c);
        __syncwarp();
        bf16* mine = solved + (row0 + group) * Plan::right_row + column0 + pair;
#pragma unroll
        for (int n = 0; n < kTiles; ++n) {
            split_two(right[0][n][0] - acc[n][0], right[0][n][1] - acc[n][1], mine + 8 * n, Plan::right_plane);
            split_two(right[0][n][2] - acc[n][2], right[0][n][3] - acc[n][3], mine + 8 * Plan::right_row + 8 * n, Plan::right_plane);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                acc[n][i] = 0.0f;
#pragma unroll
                for (int r = 0; r + 1 < kChunk / 16; ++r) right[r][n][i] = right[r + 1][n][i];  // the next block's to the first place
            }
        }
        __syncwarp();
        accumulate(inverse_at + 16 * block * Plan::inverse_row * 2, Plan::inverse_plane, row0);
#pragma unroll
        for (int n = 0; n < kTiles; ++n) fit += acc[n][0] + acc[n][1];
        __syncwarp();
        const int row = 16 * block + group;
#pragma unroll
        for (int n = 0; n < kTiles; ++n) {
            if (block + 1 < kChunk / 16) {
                split_two(acc[n][0], acc[n][1], mine + 8 * n, Plan::right_plane);
                split_two(acc[n][2], acc[n][3], mine + 8 * Plan::right_row + 8 * n, Plan::right_plane);
            }
            if (of_values) {
                float* x = args.u + (at * kChunk + row) * V + column0 + 8 * n + pair;
                store_pair(x, acc[n][0], acc[n][1]);
                store_pair(x + 8 * V, acc[n][2], acc[n][3]);
            } else {
                bf16* y = args.y + kParts * at * kChunk * kDim + turned(row, column0 - V + 8 * n + pair);  // (row + 8 is turned alike)
                split_two(acc[n][0], acc[n][1], y, kChunk * kDim);
                split_two(acc[n][2], acc[n][3], y + 8 * kDim, kChunk * kDim);
            }
        }
        __syncwarp();
    }
    // A row that is not finite has met the inverses' zeros in the earlier rows of its 16, and a thread's upper results show it: the warp's
    // columns once more by plain substitution, a lane a column.
    if (!__all_sync(0xffffffffu, isfinite(fit))) {
        const int column = column0 + (tid & 31);
        const float* from = of_values ? value_rows + column : key_rows + column - V;
        float x[kChunk];
#pragma unroll 1
        for (int i = 0; i < kChunk; ++i) {
            float sum = (of_values ? beta[i] : beta[i] * expf((float)logs[i]) * unit[i]) * (i < count ? from[(size_t)i * args.conv_stride] : 0.0f);
#pragma unroll 1
            for (int j = 0; j < i; ++j) sum = fmaf(-whole_one(matrix + i * kRow + j, kPlane), x[j], sum);
            x[i] = sum;
            if (of_values) {
                args.u[(at * kChunk + i) * V + column] = sum;
            } else {
                uint32_t hi, mid, lo;
                split_pair(sum, 0.0f, hi, mid, lo);
                unsigned short* y = reinterpret_cast<unsigned short*>(args.y + kParts * at * kChunk * kDim + turned(i, column - V));
                y[0] = (unsigned short)hi, y[kChunk * kDim] = (unsigned short)mid, y[2 * kChunk * kDim] = (unsigned short)lo;
            }
        }
    }
}

// grid (V / kColumns, heads, sequences); block kCarryThreads: a warp has 16 coordinates of S (and 16 tokens of u) at eight of the block's
// columns, as its products leave them.  The next two chunks' y and keys arrive by bulk copies, the next one's x in registers, while this one's are
// used.  (Bound by the latency of the two products one after the other.  2,048 tokens: 65 us with four warps of sixteen columns each, one to a
// scheduler, 59 with eight; 45.5 when the copies were no longer 3,072 of 16 bytes, whose issue took 850 of a chunk's 3,100 cycles.  Two and
// three chunks, where the ring's start weighs most: a layer of 128 tokens 85.3 -> 79.1 us, of 192 92.4 -> 86.3.)
constexpr int kCarryPlane = kChunk * kDim;
constexpr int kCarryStage = 2 * kParts * kCarryPlane, kCarryStages = 3;                    // y, keys
constexpr int kCarryBytes = (kCarryStages * kCarryStage + 2 * kParts * kNarrowPlane) * 2;  // and S, u

static __device__ int g_carry_status = 0;  // 1: a copy did not arrive within about two seconds

// The bounded wait for a stage: false in every thread that gave up.
__device__ __forceinline__ bool carry_wait(uint32_t bar, uint32_t parity) {
    const long long start = clock64();
    uint32_t done = 0;
    for (;;) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
            "selp.u32 %0, 1, 0, p;\n\t}"
            : "=r"(done)
            : "r"(bar), "r"(parity)
            : "memory");
        if (done) return true;
        if (clock64() - start > 4000000000LL) {
            atomicExch(&g_carry_status, 1);
            return false;
        }
    }
}

template <int V>
__global__ void __launch_bounds__(kCarryThreads)
delta_chunks_carry_kernel(const DeltaChunkArgs args) {
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) unsigned char shared[];
    __shared__ __align__(8) uint64_t arrived[kCarryStages];
    bf16* stages = reinterpret_cast<bf16*>(shared);
    bf16 *s_planes = stages + kCarryStages * kCarryStage, *u_planes = s_planes + kParts * kNarrowPlane;
    const int column0 = blockIdx.x * kColumns, head = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], tokens = args.cu_q[seq + 1] - first;
    if (tokens <= 0) return;
    const int chunks = (tokens + kChunk - 1) / kChunk;
    const int warp = (tid >> 5) & 3, tile0 = 8 * (tid >> 7), group = (tid & 31) >> 2, pair = 2 * (tid & 3);
    const int row = 16 * warp + group;             // and row + 8
    const int column = column0 + tile0 + pair;     // and the next one
    const size_t place0 = place_of(first, seq, 0);
    auto item = [&](int chunk) { return (place0 + chunk) * args.heads + head; };
    if (tid == 0) {
#pragma unroll
        for (int i = 0; i < kCarryStages; ++i) asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&arrived[i])));
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    auto fetch = [&](int chunk) {
        if (tid != 0 || chunk >= chunks) return;
        const uint32_t bar = smem_u32(&arrived[chunk % kCarryStages]), to = smem_u32(stages + chunk % kCarryStages * kCarryStage);
        constexpr uint32_t half = kParts * kCarryPlane * 2;
        const bf16 *y = args.y + kParts * item(chunk) * kChunk * kDim, *keys = args.keys + kParts * item(chunk) * kChunk * kDim;
        asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(2 * half) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to), "l"(y), "r"(half), "r"(bar) : "memory");
        asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(to + half), "l"(keys), "r"(half), "r"(bar) : "memory");
    };
    float2 x[2];
    double log_keep;
    auto fetch_x = [&](int chunk) {
        const float* from = args.u + item(chunk) * kChunk * V + column;
        x[0] = load_pair(from + (size_t)row * V);
        x[1] = load_pair(from + (size_t)(row + 8) * V);
        log_keep = args.logs[item(chunk) * kChunk + kChunk - 1];  // (made a float where it is used: that waits for it)
    };
    fetch(0);
    fetch(1);
    fetch_x(0);
    float* stored = args.state + (size_t)args.slots[seq] * args.state_stride + (size_t)head * kDim * V + column;
    float s[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) s[i] = stored[(size_t)(row + 8 * (i / 2)) * V + i % 2];
    // right operands: 32 rows at once, for two steps of 16
    const int lane = tid & 31, turn = lane & 7;
    const uint32_t right_lanes = (lane * kNarrowRow + tile0) * 2, s_at = smem_u32(s_planes) + right_lanes, u_at = smem_u32(u_planes) + right_lanes;
    // y [16 rows of the warp][k] by rows, keys [k][16 columns of the warp] by columns; units turned by the row, whose low bits are the lane's
    const uint32_t y_at = smem_u32(stages) + (16 * warp + (lane & 15)) * kDim * 2;
    const uint32_t key_at = smem_u32(stages) + kParts * kCarryPlane * 2 + ((lane >> 4) * 8 + turn) * kDim * 2 + ((2 * warp + (lane >> 3 & 1)) ^ turn) * 16;
    auto steps = [&](float (&d)[4], float scale, uint32_t left, bool keys, uint32_t right) {  // d = scale * d + left (16 x 64) . right (64 x 8)
#pragma unroll
        for (int k = 0; k < 64; k += 32) {
            uint32_t both[kParts][4];
            Parts a[2];
#pragma unroll
            for (int p = 0; p < kParts; ++p) {
                ldmatrix4_turned(both[p], right + (k * kNarrowRow + p * kNarrowPlane) * 2);
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    if (keys) ldmatrix4_turned(a[half][p], left + (p * kCarryPlane + (k + 16 * half) * kDim) * 2);
                    else ldmatrix4(a[half][p], left + p * kCarryPlane * 2 + (((k + 16 * half) / 8 + (lane >> 4)) ^ turn) * 16);
                }
            }
            const HalfParts first_half = {{both[0][0], both[0][1]}, {both[1][0], both[1][1]}, {both[2][0], both[2][1]}};
            const HalfParts second_half = {{both[0][2], both[0][3]}, {both[1][2], both[1][3]}, {both[2][2], both[2][3]}};
            split_product_twice(d, k == 0 ? scale : 1.0f, a[0], first_half, a[1], second_half);
        }
    };
    for (int chunk = 0; chunk < chunks; ++chunk) {
        float* start = args.starts + item(chunk) * kDim * V + column;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            split_two(s[2 * half], s[2 * half + 1], s_planes + (row + 8 * half) * kNarrowRow + tile0 + pair, kNarrowPlane);
            store_pair(start + (size_t)(row + 8 * half) * V, s[2 * half], s[2 * half + 1]);
        }
        const bool here = carry_wait(smem_u32(&arrived[chunk % kCarryStages]), chunk / kCarryStages & 1);
        if (!__syncthreads_and(here)) {
            // Nobody leaves while copies may still arrive, and nobody takes what was not computed for a result: the state and the starts of the
            // chunks that are left are no numbers.
            for (int later = chunk; later < min(chunks, chunk + kCarryStages - 1); ++later) carry_wait(smem_u32(&arrived[later % kCarryStages]), later / kCarryStages & 1);
            const float none = __int_as_float(0x7fffffff);
            for (int later = chunk; later < chunks; ++later)
                for (int half = 0; half < 2; ++half) store_pair(args.starts + item(later) * kDim * V + column + (size_t)(row + 8 * half) * V, none, none);
            for (int i = 0; i < 4; ++i) stored[(size_t)(row + 8 * (i / 2)) * V + i % 2] = none;
            return;
        }
        // S, y and the keys are there; nobody reads the stage before any more
        fetch(chunk + kCarryStages - 1);
        const uint32_t stage = chunk % kCarryStages * kCarryStage * 2;
        const float keep = expf((float)log_keep);
        float product[4] = {};
        steps(product, 1.0f, y_at + stage, false, s_at);
        float* to = args.u + item(chunk) * kChunk * V + column;
#pragma unroll
        for (int half = 0; half < 2; ++half) {
            const float lo = x[half].x - product[2 * half], hi = x[half].y - product[2 * half + 1];
            split_two(lo, hi, u_planes + (row + 8 * half) * kNarrowRow + tile0 + pair, kNarrowPlane);
            store_pair(to + (size_t)(row + 8 * half) * V, lo, hi);
        }
        if (chunk + 1 < chunks) fetch_x(chunk + 1);
        __syncthreads();
        steps(s, keep, key_at + stage, true, u_at);
    }
#pragma unroll
    for (int i = 0; i < 4; ++i) stored[(size_t)(row + 8 * (i / 2)) * V + i % 2] = s[i];
}

// grid (heads, most chunks of a sequence, sequences); block kResultThreads: a warp has 16 tokens and half of the V columns of their
// results (both halves' warps make the weights that they share).  u takes the start's place in shared memory, so that two blocks fit on
// a multiprocessor.
template <int V>
struct ResultPlan {
    static constexpr int wide_row = V + 8, wide_plane = 64 * wide_row;
    static constexpr int queries = 0, keys = queries + kParts * kPlane, wide = keys + kParts * kPlane, bytes = (wide + kParts * wide_plane) * 2;
};

template <typename T, int V>
__global__ void __launch_bounds__(kResultThreads, 2)
delta_chunks_results_kernel(const DeltaChunkArgs args) {
    using Plan = ResultPlan<V>;
    grid_launch_dependents();
    grid_dependency_wait();
    extern __shared__ __align__(16) unsigned char shared[];
    bf16* planes = reinterpret_cast<bf16*>(shared);
    __shared__ double logs[kChunk];
    __shared__ float square_sums[2][kChunk];
    const int head = blockIdx.x, chunk = blockIdx.y, seq = blockIdx.z, tid = threadIdx.x;
    const int first = args.cu_q[seq], count = min(kChunk, args.cu_q[seq + 1] - first - chunk * kChunk);
    if (count <= 0) return;
    const size_t token0 = (size_t)first + chunk * kChunk;
    const size_t at = place_of(first, seq, chunk) * args.heads + head;
    constexpr int kPieces = 64 * V / 8 / kResultThreads;  // eights of the start, and of u, that a thread brings
    float x[kPieces][8];
    auto ask = [&](const float* from) {
#pragma unroll
        for (int i = 0; i < kPieces; ++i) load8(from + 8 * (tid + i * kResultThreads), x[i]);
    };
    auto put = [&]() {
        float fit = 0.0f;
#pragma unroll
        for (int i = 0; i < kPieces; ++i) {
            const int piece = tid + i * kResultThreads;
            fit += fitness(x[i]);
            store_parts(planes + Plan::wide + piece / (V / 8) * Plan::wide_row + piece % (V / 8) * 8, Plan::wide_plane, x[i]);
        }
        return fit;
    };
    // everything is asked for before any of it is waited for
    const float* rows = args.conv + token0 * args.conv_stride;
    const int qk_head = head / (args.heads / args.kv_heads);
    {
        UnitRows<kResultThreads> k(rows + args.k_at + qk_head * kDim, args.conv_stride, count), q(rows + args.q_at + qk_head * kDim, args.conv_stride, count);
        if (tid < kChunk) logs[tid] = args.logs[at * kChunk + tid];
        ask(args.starts + at * kDim * V);
        k.put(count, args.unit_eps, 1.0f, planes + Plan::keys, nullptr);
        q.put(count, args.unit_eps, 0.125f, planes + Plan::queries, nullptr);  // 64^(-1/2)
        put();
    }
    __syncthreads();
    const int warp = (tid >> 5) & 3, half_columns = tid >> 7, column0 = half_columns * (V / 2), group = (tid & 31) >> 2, pair = 2 * (tid & 3);
    const uint32_t base = smem_u32(planes);
    const uint32_t query_at = base + (Plan::queries + 16 * warp * kRow) * 2 + lanes_by_row(kRow), key_at = base + Plan::keys * 2 + lanes_by_column(kRow);
    const uint32_t wide_at = base + (Plan::wide + column0) * 2 + lanes_by_row(Plan::wide_row);
    float acc[V / 16][4] = {}, weights[kChunk / 8][4] = {};
    ask(args.u + at * kChunk * V);  // (arrives while the start is multiplied)
#pragma unroll 1
    for (int d = 0; d < kDim; d += 16) {
        Parts a, b;
        load_parts(a, query_at + d * 2, kPlane);
#pragma unroll
        for (int n = 0; n < V / 16; n += 2) {  // S_0^T q
            load_parts_turned(b, wide_at + (d * Plan::wide_row + 8 * n) * 2, Plan::wide_plane);
            split_products(acc[n], acc[n + 1], a, b);
        }
    }
    __syncthreads();  // nobody reads the start any more
    const float fit = put();
#pragma unroll 1
    for (int d = 0; d < kDim; d += 16) {
        Parts a, b;
        load_parts(a, query_at + d * 2, kPlane);
#pragma unroll
        for (int n = 0; n < kChunk / 8; n += 2) {  // q . k over the tokens up to the warp's last
            if (n > 2 * warp) break;
            load_parts(b, key_at + (8 * n * kRow + d) * 2, kPlane);
            split_products(weights[n], weights[n + 1], a, b);
        }
    }
    const int row = 16 * warp + group;
    const float from_start[2] = {expf((float)logs[row]), expf((float)logs[row + 8])};
#pragma unroll
    for (int n = 0; n < V / 16; ++n)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[n][i] = __fmul_rn(acc[n][i], from_start[i / 2]);  // (rounded by itself, whatever follows)
    const bool spoiled = __syncthreads_or(!isfinite(fit));
#pragma unroll 1
    for (int n = 0; n <= 2 * warp; n += 2) {
#pragma unroll
        for (int m = 0; m < 2; ++m)
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int to = row + 8 * (i / 2), from = 8 * (n + m) + pair + i % 2;
                weights[m][i] = from <= to ? weights[m][i] * expf((float)(logs[to] - logs[from])) : 0.0f;
            }
        Parts a, b;
        split_pair(weights[0][0], weights[0][1], a[0][0], a[1][0], a[2][0]);
        split_pair(weights[0][2], weights[0][3], a[0][1], a[1][1], a[2][1]);
        split_pair(weights[1][0], weights[1][1], a[0][2], a[1][2], a[2][2]);
        split_pair(weights[1][2], weights[1][3], a[0][3], a[1][3], a[2][3]);
#pragma unroll
        for (int c = 0; c < V / 16; c += 2) {
            load_parts_turned(b, wide_at + (8 * n * Plan::wide_row + 8 * c) * 2, Plan::wide_plane);
            split_products(acc[c], acc[c + 1], a, b);
        }
        move_up<2>(weights);
    }
    if (spoiled) {  // a row of u that is not finite: see causal_products
        const bf16 *queries = planes + Plan::queries, *keys = planes + Plan::keys;
        auto weight = [&](int token, int from) { return whole_dot<kDim>(queries + token * kRow, keys + from * kRow, kPlane) * expf((float)(logs[token] - logs[from])); };
        start_products<kDim>(acc, queries + row * kRow, kRow, kPlane, args.starts + at * kDim * V + column0 + pair, V);
#pragma unroll
        for (int n = 0; n < V / 16; ++n)
#pragma unroll
            for (int i = 0; i < 4; ++i) acc[n][i] *= from_start[i / 2];
        causal_products(acc, row, weight, planes + Plan::wide + column0 + pair, Plan::wide_row, Plan::wide_plane);
    }
    // norm, gain and gate: a row's V results lie with four neighbouring lanes of two warps.  Gates and gains are asked for at once, before the
    // sums: one after another, each behind a store and a division, they were 20,000 of a block's 52,000 cycles.
    const size_t column = (size_t)head * V + column0 + pair;
    Pair<T> gates[2][V / 16];
    float2 gain[V / 16];
#pragma unroll
    for (int n = 0; n < V / 16; ++n) {
        gain[n] = load_pair(args.gain + column0 + 8 * n + pair);
#pragma unroll
        for (int half = 0; half < 2; ++half)  // (rows beyond the chunk's last: that one's, and not used)
            gates[half][n] = *reinterpret_cast<const Pair<T>*>((const T*)args.gate_in + (token0 + min(row + 8 * half, count - 1)) * args.in_stride + column + 8 * n);
    }
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
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        const int to = row + 8 * half;
        if (to >= count) continue;
        const float inv = args.out_scale / sqrtf((square_sums[0][to] + square_sums[1][to]) / (float)V + args.eps);
        T* dst = (T*)args.out + (token0 + to) * args.out_stride + column;
        float open[V / 8];
#pragma unroll
        for (int n = 0; n < V / 16; ++n) {
            const float2 z = load_pair(reinterpret_cast<const T*>(&gates[half][n]));
            open[2 * n] = z.x, open[2 * n + 1] = z.y;
        }
        sigmoids(open);
#pragma unroll
        for (int n = 0; n < V / 16; ++n) {
            const float2 z = load_pair(reinterpret_cast<const T*>(&gates[half][n]));
            store_pair(dst + 8 * n, acc[n][2 * half] * inv * gain[n].x * (z.x * open[2 * n]), acc[n][2 * half + 1] * inv * gain[n].y * (z.y * open[2 * n + 1]));
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
    constexpr int solve = SolvePlan<V>::bytes, results = ResultPlan<V>::bytes;
    if (int status = reserve(delta_chunks_solve_kernel<T, V>, solve)) return status;
    if (int status = reserve(delta_chunks_carry_kernel<V>, kCarryBytes)) return status;
    if (int status = reserve(delta_chunks_results_kernel<T, V>, results)) return status;
    const dim3 grid(args.heads, chunks, sequences);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_solve_kernel<T, V>), grid, dim3(SolvePlan<V>::threads), solve, stream, true, args);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_carry_kernel<V>), dim3(V / kColumns, args.heads, sequences), dim3(kCarryThreads), kCarryBytes, stream, true,
              args);
    MB_LAUNCH("gated_delta_chunks", (delta_chunks_results_kernel<T, V>), grid, dim3(kResultThreads), results, stream, true, args);
    return check_launch("gated_delta_chunks");
}

}  // namespace mb

using namespace mb;

// Arguments as mb_gated_delta_scan's, with key heads of 64 numbers and value heads of 64 or 128; conv is only read.  scratch: floats,
// (places * heads) * (2 * 64 * vdim + 3 * 64 * 64 + 128), 16-byte aligned, with places = tokens / 64 + sequences.
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
    args.y = reinterpret_cast<bf16*>(args.starts + items * kDim * vdim);
    args.keys = args.y + kParts * items * kChunk * kDim;
    args.logs = reinterpret_cast<double*>(args.keys + kParts * items * kChunk * kDim);
    if (dtype == MB_F32) return vdim == 64 ? launch_chunks<float, 64>(args, sequences, chunks, stream) : launch_chunks<float, 128>(args, sequences, chunks, stream);
    if (dtype == MB_BF16)
        return vdim == 64 ? launch_chunks<__nv_bfloat16, 64>(args, sequences, chunks, stream) : launch_chunks<__nv_bfloat16, 128>(args, sequences, chunks, stream);
    return fail("gated_delta_chunks: unknown dtype code %d", dtype);
}

// 0 while no wait for a copy ever gave up.
MB_EXPORT int mb_gated_delta_chunks_status() {
    int status = 0;
    if (cudaMemcpyFromSymbol(&status, g_carry_status, sizeof(int)) != cudaSuccess) return -1;
    return status;
}
