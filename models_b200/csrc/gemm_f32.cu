// 32-bit matrix product on the fifth-generation tensor cores: C[M, N] = A[M, K] . W[N, K]^T of floats, whose 24 bits are all
// multiplied.  It is the matrix product of the 32-bit path of the whole model.
//
// out[r] = sum_c W[r, c] * x[c] (integrallis/models, backend-java/.../ops/TensorOps.java:61-63).
// A float is the sum of three bfloat16 numbers (float_parts.cuh), and a product of floats that of six products of these (the other
// three are 2^-24 of it at most: a second part is up to 2^-8 of its float, a third up to 2^-17), summed in float:
//   * the products of the two roundings, 64 columns of K at a time, in tensor memory, and these sums by float additions in
//     registers: a tensor core cuts its sum off where a float addition rounds, so no long sum may stay there;
//   * the five smaller products, 2^-7 of the whole together, in tensor memory over all of the block's columns: the cut takes up to
//     2^-31 K of the whole from them (20 steps a stage, 2^-23 of their sum each).
// Every result is the sum, in order, of up to four such sums over consecutive parts of K; the parts follow from N and K alone, and
// every call runs the same operations on a row, so a row's result depends neither on the other rows of the call, nor on where it
// sits in a tile, nor on alignment, nor on which of the kernels below computes it.
//
// Off the sums in 64 bits by 1.0e-7 to 1.4e-7 (2-norm; K 2,048 and 8,192); chains of FMAs over the same parts were 2.9e-7 to 5.8e-7 off.
// 301 rows, W of 16,384 x 2,048 that are bfloat16 numbers: 89 us, 2,048 x 8,192 52 us, 3,072 x 2,048 37 us, 2,048 x 2,048 21 us (whole
// floats 104, 62, 41 and 24); FMAs on 8 x 8 results a thread took 480, 274, 114 and 80 us, at 46 of the CUDA cores' 74 TFLOP/s.
// From 33 rows on a block is bound by the splitting of W; the kernel for few rows says what bounds it.
//
// 128 rows of W are the products' first operand and up to 160 rows of A the second.  Eight warps bring W from memory (loads of the
// next columns are under way while these are worked on) and split it into shared memory, one brings A, which a kernel before has
// split (of few rows, and in small products, the eight warps split it too: in 301 rows that doubled their work, 127 us for 92), one issues the products,
// and four hold the sums, a row of W per thread.  Weights that are bfloat16 numbers -- most models' are, in the 32-bit mode too -- have
// two parts of zeros, whose products are left out: each stage of W says whether it is such.
//
// Both operands are split times 2^24, and the sums divided by 2^48: the parts of every float are whole then, also where it is so small that
// bfloat16 would have no bits left for its third.  Sums that are not finite -- a float was not, or was above 2^103, or the result is above
// 2^79 -- are computed anew from the floats, in the order of K: no other row of A or W sees such a float.  (Results decide, and not
// operands, so that every kernel below decides alike.)
#include "tcgen05.cuh"
#include "float_parts.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace cg = cooperative_groups;

MB_DEFINE_LAST_ERROR()

namespace mb {

constexpr int kTileN = 128;           // rows of the products' first operand: a block's rows of W, or twice as many
constexpr int kChunk = 64;            // columns of K per stage: a row of 128 bytes of bfloat16
constexpr int kAdders = 4, kSplitters = 8;  // warps; after them one issues products and one brings A (two keep their warpgroup company)
constexpr int kIssuer = kAdders + kSplitters, kBringer = kIssuer + 1;
constexpr int kThreads = 32 * (kAdders + kSplitters + 4);
constexpr int kRegisters = 128;       // a thread's at launch; the warpgroups trade them once (what is in flight to a register that is given back would be lost)
constexpr int kPlaneW = kTileN * 128;
constexpr int kPlaneA = 32 * 128;     // times NB
constexpr int kMaxStages = 3;
constexpr int kInlineRows = 32;       // most rows of A that are split where they are multiplied
constexpr int kSlabRows = 2048;       // rows of A that are split at a time
constexpr uint64_t kUp = 0x4b8000004b800000ull, kDown = 0x2780000027800000ull;  // pairs of 2^24, times which both operands are split, and of 2^-48

// NB: 32 rows of A each.  kRowsW: rows of W per block (64 leave half of the products' first operand to chance, unread).
template <int NB, int kRowsW>
struct Plan {
    static constexpr bool kInline = NB == 1;
    static constexpr int kRows = 32 * NB;
    static constexpr int kStageBytes = 3 * (kPlaneW + NB * kPlaneA);
    static constexpr int kStages = NB <= 2 ? 3 : 2;
    static constexpr int kBytes = kStages * kStageBytes + 1024;
    static constexpr int kColumns = 3 * kRows <= 128 ? 128 : 3 * kRows <= 256 ? 256 : 512;  // of tensor memory: two sums, and the smaller products'
    // Registers a thread: shares of the four warpgroups' 128 a thread at launch.
    static constexpr int kAdderRegisters = kInline ? 80 : 224, kSplitterRegisters = kInline ? 152 : 112, kIssuerRegisters = 48;
    static_assert(kAdderRegisters + 2 * kSplitterRegisters + kIssuerRegisters <= 4 * kRegisters && kThreads == 512, "the warpgroups' shares");
    static_assert(kStages <= kMaxStages && kStages * kStageBytes >= kRows * kRowsW * 4, "the parts' sums take the place of the stages");
};

// A thread's eight of a row's 64 columns, as four pairs: four columns from `from` and the four 32 further (so that eight threads' loads
// cover whole lines); `left` columns are left from `from` on, and none is wanted of a stage that is not there.  They stand side by side in
// the stage: both operands have the same order of K there.  kEven: whole 16-byte pieces, by loads that a predicate holds back (pieces
// behind the last column are left as they are); else column by column, zeros behind the last.  (Plain loads: the kernel before may just have written the row.)
template <bool kEven>
__device__ __forceinline__ void load_eight(uint64_t (&v)[4], const float* from, int left, bool wanted) {
    if (kEven) {
        asm volatile(
            "{\n\t.reg .pred p, q;\n\t"
            "setp.gt.s32 p, %5, 0;\n\t"
            "setp.gt.s32 q, %5, 32;\n\t"
            "@p ld.global.v2.b64 {%0, %1}, [%4];\n\t"
            "@q ld.global.v2.b64 {%2, %3}, [%4 + 128];\n\t}"
            : "+l"(v[0]), "+l"(v[1]), "+l"(v[2]), "+l"(v[3])
            : "l"(from), "r"(left)
            : "memory");
    } else if (wanted) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int column = 2 * (j % 2) + j / 2 * 32;
            v[j] = pair_of(column < left ? from[column] : 0.0f, column + 1 < left ? from[column + 1] : 0.0f);
        }
    }
}

// Four neighbouring columns, as two pairs, in the same way.
template <bool kEven>
__device__ __forceinline__ void load_four(uint64_t (&v)[2], const float* from, int left) {
    if (kEven) {
        asm volatile(
            "{\n\t.reg .pred p;\n\t"
            "setp.gt.s32 p, %3, 0;\n\t"
            "@p ld.global.v2.b64 {%0, %1}, [%2];\n\t}"
            : "+l"(v[0]), "+l"(v[1])
            : "l"(from), "r"(left)
            : "memory");
    } else {
        v[0] = pair_of(0 < left ? from[0] : 0.0f, 1 < left ? from[1] : 0.0f);
        v[1] = pair_of(2 < left ? from[2] : 0.0f, 3 < left ? from[3] : 0.0f);
    }
}

// Their parts, 16 bytes to each of three planes; `smaller` gathers the bits of the two smaller ones.
__device__ __forceinline__ void split_eight(const uint64_t (&v)[4], unsigned char* at, size_t plane_bytes, uint32_t& smaller) {
    uint4 hi, mid, lo;
    split_pair(pair_mul(v[0], kUp), hi.x, mid.x, lo.x);
    split_pair(pair_mul(v[1], kUp), hi.y, mid.y, lo.y);
    split_pair(pair_mul(v[2], kUp), hi.z, mid.z, lo.z);
    split_pair(pair_mul(v[3], kUp), hi.w, mid.w, lo.w);
    *reinterpret_cast<uint4*>(at) = hi;
    *reinterpret_cast<uint4*>(at + plane_bytes) = mid;
    *reinterpret_cast<uint4*>(at + 2 * plane_bytes) = lo;
    smaller |= mid.x | mid.y | mid.z | mid.w | lo.x | lo.y | lo.z | lo.w;
}

__device__ __forceinline__ uint32_t elect_one() {
    uint32_t elected;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(elected));
    return elected;
}

// One step of 16 columns: to (+)= a . b.  (Whether it adds is known where it is written, and no lane is masked: a step is issued in
// half the time that umma() takes, and few rows of A are bound by the issue.)
template <bool kAdds>
__device__ __forceinline__ void issue_step(uint32_t to, uint64_t a_desc, uint64_t b_desc, uint32_t instruction) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(to), "l"(a_desc), "l"(b_desc), "r"(instruction), "n"(kAdds ? 1 : 0)
        : "memory");
}

struct FloatArgs {
    const float* a;
    const float* w;
    float* c;
    int lda, ldw, ldc, m, n, k;
    int parts, part_length;       // blocks of a cluster that share K; columns of each, a multiple of kChunk
    int weights_ready;            // W depends on no kernel that may still be running: it is asked for before the wait for the one before
};

// A, split: planes [3][m][chunks * 64], a chunk's columns in the order of load_eight, zeros behind the last.  32 chunks of rows a block.
template <bool kEven>
__global__ void __launch_bounds__(256)
split_rows_kernel(const float* __restrict__ a, int lda, int m, int k, int chunks, unsigned char* planes) {
    grid_launch_dependents();
    grid_dependency_wait();
    const size_t item = (size_t)blockIdx.x * 32 + (threadIdx.x >> 3);
    if (item >= (size_t)m * chunks) return;
    const int row = (int)(item / chunks), chunk = (int)(item % chunks), unit = threadIdx.x & 7;
    uint64_t v[4] = {};
    load_eight<kEven>(v, a + (size_t)row * lda + chunk * kChunk + 4 * unit, k - chunk * kChunk - 4 * unit, true);
    uint32_t smaller = 0;
    split_eight(v, planes + item * 128 + unit * 16, (size_t)m * chunks * 128, smaller);
}

// grid: parts of K fastest, then the tiles of A, then those of W (so that neighbours share a tile of W).
template <int NB, int kRowsW, bool kEven>
__global__ void __launch_bounds__(kThreads, 1)
gemm_f32_kernel(const __grid_constant__ CUtensorMap map_a, const FloatArgs args) {
    using P = Plan<NB, kRowsW>;
    constexpr int kPlane = NB * kPlaneA;
    constexpr int kPassesW = kRowsW / 16, kPassesA = P::kInline ? 2 * NB : 0, kHeldA = P::kInline ? 2 * NB : 1;
    constexpr uint32_t kInstruction = instruction_descriptor(kTileN, P::kRows);
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~(uintptr_t)1023);
    __shared__ __align__(8) uint64_t barriers[2 * kMaxStages + 5];
    __shared__ uint32_t tmem_base_slot;
    __shared__ int whole[kMaxStages];  // one more than the last chunk whose floats of W, in this stage, have parts beyond the first
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full_bar = smem_u32(&barriers[0]), empty_bar = smem_u32(&barriers[kMaxStages]);
    const uint32_t sum_full_bar = smem_u32(&barriers[2 * kMaxStages]), sum_empty_bar = sum_full_bar + 16, done_bar = sum_full_bar + 32;
    const int part = blockIdx.x % args.parts, tile = blockIdx.x / args.parts;
    const int a_tiles = (args.m + P::kRows - 1) / P::kRows;
    const int row0 = (tile % a_tiles) * P::kRows, col0 = (tile / a_tiles) * kRowsW;
    const int k_begin = part * args.part_length, k_end = min(args.k, k_begin + args.part_length);
    const int chunks = (k_end - k_begin + kChunk - 1) / kChunk;  // (no part is empty)

    if (threadIdx.x == 0) {
        for (int s = 0; s < P::kStages; ++s) {
            mbar_init(full_bar + 8 * s, kSplitters / 2 + (P::kInline ? 0 : 1));
            mbar_init(empty_bar + 8 * s, 1);
            whole[s] = 0;
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(sum_full_bar + 8 * b, 1);
            mbar_init(sum_empty_bar + 8 * b, kAdders);
        }
        mbar_init(done_bar, 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == kIssuer) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_base_slot)), "n"(P::kColumns));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::);
    }
    tcgen05_fence_before();
    __syncthreads();
    tcgen05_fence_after();
    const uint32_t tmem_sum = tmem_base_slot, tmem_small = tmem_sum + 2 * P::kRows;  // two sums, taken in turn by the chunks
    grid_launch_dependents();
    float* sums = reinterpret_cast<float*>(smem);

    if (warp < kAdders) {
        // ------------------------------------------------------------------ add
        if (P::kAdderRegisters > kRegisters) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::kAdderRegisters));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kAdderRegisters));
        grid_dependency_wait();
        uint64_t sum[P::kRows / 2];  // of this thread's row of W, in pairs
#pragma unroll
        for (int j = 0; j < P::kRows / 2; ++j) sum[j] = 0;
        const uint32_t lanes = (uint32_t)(warp * 32) << 16;
        bool ok = true;
        auto add = [&](uint32_t from) {
#pragma unroll
            for (int i = 0; i < P::kRows; i += 32) {
                float v[32];
                tmem_load_32_issue(from + lanes + i, v);
                tmem_load_wait();
#pragma unroll
                for (int j = 0; j < 16; ++j) sum[i / 2 + j] = pair_add(sum[i / 2 + j], pair_of(v[2 * j], v[2 * j + 1]));
            }
        };
        for (int chunk = 0; chunk < chunks && ok; ++chunk) {  // what the tensor cores summed over a chunk
            const int b = chunk & 1;
            ok = __all_sync(0xffffffffu, mbar_wait(sum_full_bar + 8 * b, chunk >> 1 & 1, 4));
            tcgen05_fence_after();
            if (ok) add(tmem_sum + b * P::kRows);
            tcgen05_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(sum_empty_bar + 8 * b);
        }
        ok = ok && __all_sync(0xffffffffu, mbar_wait(done_bar, 0, 5));
        tcgen05_fence_after();
        if (ok) add(tmem_small);
        tcgen05_fence_before();
#pragma unroll
        for (int j = 0; j < P::kRows / 2; ++j) sum[j] = ok ? pair_mul(sum[j], kDown) : ~0ull;  // (NaN, where a wait gave up: computed anew)
        // To the result, or, as one of several parts, to shared memory (every product has read the stages): [rows of A][kRowsW].
        const int col = col0 + (int)threadIdx.x;
        const int rows = (int)threadIdx.x >= kRowsW ? 0 : args.parts > 1 ? P::kRows : col < args.n ? min(P::kRows, args.m - row0) : 0;
        float* to = args.parts > 1 ? sums + threadIdx.x : args.c + (size_t)row0 * args.ldc + col;
        const size_t step = args.parts > 1 ? kRowsW : args.ldc;
#pragma unroll
        for (int j = 0; j < P::kRows; ++j)
            if (j < rows) to[j * step] = j % 2 ? high_of(sum[j / 2]) : low_of(sum[j / 2]);
        uint64_t finite = 0;  // 0, 0 or NaN
#pragma unroll
        for (int j = 0; j < P::kRows / 2; ++j) finite = pair_fma(sum[j], 0, finite);
        if (low_of(finite) + high_of(finite) != 0.0f && (int)threadIdx.x < kRowsW && col < args.n) {
#pragma unroll 1
            for (int j = 0; j < min(P::kRows, args.m - row0); ++j)
                if (!isfinite(to[j * step])) {
                    const float *a = args.a + (size_t)(row0 + j) * args.lda, *w = args.w + (size_t)col * args.ldw;
                    float total = 0.0f;
#pragma unroll 1
                    for (int k = k_begin; k < k_end; ++k) total = fmaf(a[k], w[k], total);
                    to[j * step] = total;
                }
        }
        __syncwarp();
        if (args.parts > 1) {
            cluster_sync_all();
            cluster_leave_together();
        }
    } else if (warp < kAdders + kSplitters) {
        // ------------------------------------------------------------------ bring and split
        if (P::kSplitterRegisters > kRegisters) asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(P::kSplitterRegisters));
        else asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kSplitterRegisters));
        // Two groups of four warps take the chunks in turn, so that one splits while the other waits.  Eight threads bring a row's
        // 64 columns, a group 16 rows a pass; a pass's registers take the group's next chunk as soon as they have been split.
        const int group = (warp - kAdders) / (kSplitters / 2);
        const int my_row = (threadIdx.x & 127) >> 3, unit = threadIdx.x & 7;
        uint64_t w_next[kPassesW][4] = {}, a_next[kHeldA][4] = {};
        // Rows beyond the last repeat it; nobody reads what becomes of them.  Columns beyond the last are zeros in A, and in W zeros or
        // what a load before left: floats of the same row, which zeros leave without a trace unless one of them is not finite, and then
        // the row's results are not either.
        const float* w_from = args.w + (size_t)col0 * args.ldw + k_begin + 4 * unit;
        const float* a_from = args.a + (size_t)row0 * args.lda + k_begin + 4 * unit;
        const int w_last = args.n - 1 - col0, a_last = args.m - 1 - row0;
        auto fetch_w = [&](int wanted, int p) {
            const int at = wanted * kChunk;
            load_eight<kEven>(w_next[p], w_from + (at + (long long)min(16 * p + my_row, w_last) * args.ldw), k_end - k_begin - at - 4 * unit, wanted < chunks);
        };
        auto fetch_a = [&](int wanted, int p) {
            const int at = wanted * kChunk;
            const int left = k_end - k_begin - at - 4 * unit;
            if (kEven && left < 36) a_next[p][2] = a_next[p][3] = 0;
            if (kEven && left <= 0) a_next[p][0] = a_next[p][1] = 0;
            load_eight<kEven>(a_next[p], a_from + (at + (long long)min(16 * p + my_row, a_last) * args.lda), left, wanted < chunks);
        };
        if (!args.weights_ready) grid_dependency_wait();
#pragma unroll
        for (int p = 0; p < kPassesW; ++p) fetch_w(group, p);
        grid_dependency_wait();
#pragma unroll
        for (int p = 0; p < kPassesA; ++p) fetch_a(group, p);
        bool ok = true;
        for (int chunk = group; chunk < chunks && ok; chunk += 2) {
            const int stage = chunk % P::kStages;
            ok = __all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * stage, (chunk / P::kStages & 1) ^ 1, 1));  // (a stage starts free)
            if (!ok) break;
            unsigned char* at = smem + stage * P::kStageBytes + my_row * 128 + ((unit ^ (my_row & 7)) << 4);  // the 128-byte swizzle
            uint32_t smaller = 0, nothing = 0;
#pragma unroll
            for (int p = 0; p < kPassesW; ++p) {
                split_eight(w_next[p], at + p * 2048, kPlaneW, smaller);
                fetch_w(chunk + 2, p);
            }
#pragma unroll
            for (int p = 0; p < kPassesA; ++p) {
                split_eight(a_next[p], at + 3 * kPlaneW + p * 2048, kPlane, nothing);
                fetch_a(chunk + 2, p);
            }
            if ((smaller & 0x7fff7fffu) != 0) whole[stage] = chunk + 1;
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
            __syncwarp();
            if (lane == 0) mbar_arrive(full_bar + 8 * stage);
        }
        __syncwarp();
        if (args.parts > 1) {  // the cluster's blocks share the rows and add the parts in their order
            cluster_sync_all();
            for (int i = threadIdx.x - 32 * kAdders; i < P::kRows / args.parts * (kRowsW / 4); i += 32 * kSplitters) {  // (parts is 2 or 4)
                const int r = i / (kRowsW / 4) * args.parts + part, piece = i % (kRowsW / 4) * 4;
                const int row = row0 + r, col = col0 + piece;
                if (row >= args.m || col >= args.n) continue;
                float4 v[4];
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p < args.parts) v[p] = *reinterpret_cast<const float4*>(cg::this_cluster().map_shared_rank(sums, p) + r * kRowsW + piece);
                float4 total = v[0];
#pragma unroll
                for (int p = 1; p < 4; ++p)
                    if (p < args.parts) total.x += v[p].x, total.y += v[p].y, total.z += v[p].z, total.w += v[p].w;
                float* to = args.c + (size_t)row * args.ldc + col;
                const float out[4] = {total.x, total.y, total.z, total.w};
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (col + e < args.n) to[e] = out[e];
            }
            cluster_leave_together();  // the others read this block's sums
        }
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(P::kIssuerRegisters));
        if (warp == kIssuer) {
            // -------------------------------------------------------------- products (the warp walks together, one thread issues)
            const uint32_t elected = elect_one();
            int stage = 0;
            uint32_t phase = 0;
            for (int chunk = 0; chunk < chunks; ++chunk) {
                // The lanes wait together: one that fell behind by two passes over the stages would wait for the wrong one.
                const int b = chunk & 1;
                if (!__all_sync(0xffffffffu, mbar_wait(full_bar + 8 * stage, phase, 2))) break;
                tcgen05_fence_after();
                const uint32_t w_at = smem_u32(smem) + stage * P::kStageBytes, a_at = w_at + 3 * kPlaneW;
                const uint64_t w_desc = umma_descriptor(w_at), a_desc = umma_descriptor(a_at);
                const bool all_parts = *reinterpret_cast<volatile int*>(&whole[stage]) == chunk + 1;
                auto products = [&](int w_part, int a_part, uint32_t to, bool fresh) {
#pragma unroll
                    for (int ks = 0; ks < kChunk / 16; ++ks) {
                        const uint64_t w_step = w_desc + ((w_part * kPlaneW >> 4) + 2 * ks), a_step = a_desc + ((a_part * kPlane >> 4) + 2 * ks);
                        if (fresh && ks == 0) issue_step<false>(to, w_step, a_step, kInstruction);
                        else issue_step<true>(to, w_step, a_step, kInstruction);
                    }
                };
                if (elected) {
                    products(0, 2, tmem_small, chunk == 0);
                    if (all_parts) {
                        products(1, 1, tmem_small, false);
                        products(2, 0, tmem_small, false);
                    }
                    products(0, 1, tmem_small, false);
                    if (all_parts) products(1, 0, tmem_small, false);
                }
                // the chunk before the last has been added
                if (chunk > 1 && !__all_sync(0xffffffffu, mbar_wait(sum_empty_bar + 8 * b, (chunk >> 1 & 1) ^ 1, 3))) break;
                tcgen05_fence_after();
                if (elected) {
                    products(0, 0, tmem_sum + b * P::kRows, true);
                    umma_commit(sum_full_bar + 8 * b);
                    umma_commit(empty_bar + 8 * stage);
                }
                if (++stage == P::kStages) stage = 0, phase ^= 1;
            }
            if (elected) umma_commit(done_bar);
        } else if (warp == kBringer && !P::kInline) {
            // -------------------------------------------------------------- A's parts
            grid_dependency_wait();
            const uint32_t elected = elect_one();
            int stage = 0;
            uint32_t phase = 1;
            for (int chunk = 0; chunk < chunks; ++chunk) {
                if (!__all_sync(0xffffffffu, mbar_wait(empty_bar + 8 * stage, phase, 6))) break;
                if (elected) {
                    mbar_expect_tx(full_bar + 8 * stage, 3 * kPlane);
                    const uint32_t to = smem_u32(smem) + stage * P::kStageBytes + 3 * kPlaneW;
#pragma unroll
                    for (int p = 0; p < 3; ++p) tma_load_2d(to + p * kPlane, &map_a, k_begin + chunk * kChunk, p * args.m + row0, full_bar + 8 * stage);
                }
                if (++stage == P::kStages) stage = 0, phase ^= 1;
            }
        }
        __syncwarp();
        if (args.parts > 1) {
            cluster_sync_all();
            cluster_leave_together();
        }
    }
    __syncthreads();
    if (warp == kIssuer) {
        tcgen05_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem_sum), "n"(P::kColumns));
    }
}

// ---- Up to eight rows of A: the weights' stream bounds the product.  A warp owns sixteen rows of W and copies them to shared memory in
// whole lines, kStages - 1 chunks ahead, in a ring of its own; its lanes split them and multiply them by mma.sync, whose sums over 16
// columns are the tcgen05 ones, bit by bit, in whatever order these columns stand: the same steps in the same order give the same results.
// A's parts lie in shared memory, split by the block itself.
// Bound, over long rows, by what a warp does with a chunk, 3.5 to 7 warps to a multiprocessor, else by the stream (268 MB at 5.5 TB/s).
// One row, us, W of bfloat16 numbers and of floats (before that as chains of float FMAs): 2,048 x 2,048 6.7 and 7.7 (6.5), 3,072 x 2,048 8.1
// and 9.4 (7.7), 2,048 x 8,192 17.3 and 21.8 (17.0), 4,096 x 4,096 14.0 and 16.7 (16.2), 16,384 x 2,048 25.5 and 28.3 (30.5), 32,768 x 2,048
// 48.9 and 47 (52).  Chunks in registers, 16 bytes of a row to a lane, took 7.5, 8.9, 22.6, 17, 30.4 and 57.6; smaller parts made of
// weights that have none 7.5, 8.9, 21.8, 16.9, 29.4 and 50.1; tiles of eight rows, the instruction's other eight zeros, 6.8, 7.9, 18.4, 16.3
// and, of 4,096 x 4,096 floats, 20.2.
constexpr int kFewRows = 8, kFewTile = 16, kFewMostWarps = 16;
constexpr int kFewBytes = 216 * 1024;  // most shared memory that a block asks for
constexpr int kFewChunkBytes = kFewTile * kChunk * (int)sizeof(float);
constexpr int kFewBatch = 4;           // a thread's loads of A that are under way together
// A's parts: [row][chunk][16 columns][3 parts][4 lanes] pairs of words (a lane's two operand registers); rows lie a few words apart from
// whole lines, so that the lanes of different rows meet different banks.
__host__ __device__ constexpr int few_row(int chunks) { return chunks * 48 + 4; }

__device__ __forceinline__ void mma_step(float (&d)[4], const uint32_t (&a)[4], uint2 b) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b.x), "r"(b.y));
}
// Four neighbouring columns, zeros behind the last.
template <bool kEven>
__device__ __forceinline__ void copy_four(uint32_t to, const float* from, int left) {
    if (kEven) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(to), "l"(left > 0 ? from : from + left - 4), "r"(left > 0 ? 16 : 0) : "memory");
    } else {
#pragma unroll
        for (int e = 0; e < 4; ++e)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(to + 4 * e), "l"(e < left ? from + e : from + left - 1), "r"(e < left ? 4 : 0) : "memory");
    }
}
// Where 16-byte piece `piece` of a row's chunk lies: what eight lanes read together (two rows, pieces 0, 1, 8 and 9 from an even one on) and
// what they copy together (eight pieces of a row) meet all banks.
__device__ __forceinline__ int few_place(int row, int piece) { return row * 256 + (piece >> 3) * 128 + (((piece & 7) ^ (piece >> 3) * 2 ^ (row & 1) * 4) << 4); }

// One part of K: a block's warps take tiles of W in turn.  Several: a warp takes one tile, and the part's cluster rank is blockIdx.x % parts.
template <bool kEven, int kStages>
__global__ void __launch_bounds__(32 * kFewMostWarps)
gemm_f32_few_kernel(const FloatArgs args) {
    extern __shared__ __align__(16) uint2 few_parts[];
    __shared__ float sums[kFewRows][kFewTile * kFewMostWarps];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, group = lane >> 2, quad = lane & 3, threads = blockDim.x, warps = threads >> 5;
    const int part = blockIdx.x % args.parts, block = blockIdx.x / args.parts;
    const int k_begin = part * args.part_length, columns = min(args.k - k_begin, args.part_length);
    const int chunks = (columns + kChunk - 1) / kChunk, m = args.m, row_pairs = few_row(chunks);
    const int tiles = (args.n + kFewTile - 1) / kFewTile;
    const int first_tile = args.parts > 1 ? block * warps + warp : warp * gridDim.x + block, stride = args.parts > 1 ? tiles : warps * gridDim.x;
    grid_launch_dependents();

    unsigned char* ring = reinterpret_cast<unsigned char*>(few_parts + m * few_row(args.part_length / kChunk)) + warp * (kStages * kFewChunkBytes);
    const int piece = lane & 15;  // what the lane copies: two rows at a time
    const uint32_t put_at = (uint32_t)__cvta_generic_to_shared(ring) + few_place(lane >> 4, piece);
    const float* from[kFewTile / 2];
    int next_tile = first_tile, next_chunk = 0, next_slot = 0;
    auto begin_tile = [&]() {  // rows beyond the last repeat it
#pragma unroll
        for (int i = 0; i < kFewTile / 2; ++i) from[i] = args.w + (size_t)min(next_tile * kFewTile + 2 * i + (lane >> 4), args.n - 1) * args.ldw + k_begin + 4 * piece;
    };
    auto fetch = [&]() {
        if (next_tile < tiles) {
            const int left = columns - next_chunk * kChunk - 4 * piece;
#pragma unroll
            for (int i = 0; i < kFewTile / 2; ++i) {
                copy_four<kEven>(put_at + next_slot * kFewChunkBytes + i * few_place(2, 0), from[i], left);
                from[i] += kChunk;
            }
            if (++next_chunk == chunks) {
                next_chunk = 0, next_tile += stride;
                begin_tile();
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
        if (++next_slot == kStages) next_slot = 0;
    };
    begin_tile();
    if (!args.weights_ready) grid_dependency_wait();
#pragma unroll
    for (int i = 0; i < kStages - 1; ++i) fetch();
    grid_dependency_wait();
    // A's parts: a thread takes the four columns of one lane of a step, from 8 * step + 4 * (quad & 1) + 32 * (quad >> 1)
    const int items = chunks * 16;
    for (int first = threadIdx.x; first < m * items; first += kFewBatch * threads) {
        uint64_t v[kFewBatch][2] = {};
#pragma unroll
        for (int b = 0; b < kFewBatch; ++b) {
            const int i = first + b * threads, r = i / items, item = i - r * items, q = item & 3;
            const int at = (item >> 4) * kChunk + 8 * (item >> 2 & 3) + 4 * (q & 1) + 32 * (q >> 1);
            if (r < m) load_four<kEven>(v[b], args.a + (size_t)r * args.lda + k_begin + at, columns - at);
        }
#pragma unroll
        for (int b = 0; b < kFewBatch; ++b) {
            const int i = first + b * threads, r = i / items, item = i - r * items;
            if (r >= m) break;
            uint2 hi, mid, lo;
            split_pair(pair_mul(v[b][0], kUp), hi.x, mid.x, lo.x);
            split_pair(pair_mul(v[b][1], kUp), hi.y, mid.y, lo.y);
            uint2* to = few_parts + r * row_pairs + (item >> 2) * 12 + (item & 3);
            to[0] = hi, to[4] = mid, to[8] = lo;
        }
    }
    __syncthreads();

    const uint2* mine = few_parts + min(group, m - 1) * row_pairs + quad;  // (nobody reads the results of rows beyond the last)
    int slot = 0;
#pragma unroll 1
    for (int tile = first_tile; tile < tiles; tile += stride) {
        float sum[4] = {}, small[4] = {};  // rows group and group + 8 of W with rows 2 * quad and 2 * quad + 1 of A
#pragma unroll 1
        for (int chunk = 0; chunk < chunks; ++chunk) {
            asm volatile("cp.async.wait_group %0;" ::"n"(kStages - 2) : "memory");
            __syncwarp();  // the chunk is there for every lane, and every lane has read the one before
            uint32_t w[4][3][4] = {};  // [step][part][operand registers: row and row + 8 of the first two columns, then of the others]
            uint64_t rest[4][4];  // what their roundings leave
            uint64_t any = 0;
            const unsigned char* at = ring + slot * kFewChunkBytes;
#pragma unroll
            for (int step = 0; step < 4; ++step)
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const float4 x = *reinterpret_cast<const float4*>(at + few_place(group + 8 * h, (quad & 1) + 8 * (quad >> 1) + 2 * step));
#pragma unroll
                    for (int e = 0; e < 2; ++e) {
                        const uint64_t v = pair_mul(e == 0 ? pair_of(x.x, x.y) : pair_of(x.z, x.w), kUp);
                        w[step][0][2 * e + h] = round_pair(v);
                        rest[step][2 * e + h] = minus_rounding(v, w[step][0][2 * e + h]);
                        any |= rest[step][2 * e + h];
                    }
                }
            fetch();  // to the place of the chunk before
            if (++slot == kStages) slot = 0;
            const bool all_parts = __any_sync(0xffffffffu, any != 0);
            auto products = [&](int w_part, int a_part, float (&to)[4]) {
#pragma unroll
                for (int step = 0; step < 4; ++step) mma_step(to, w[step][w_part], mine[(chunk * 4 + step) * 12 + a_part * 4]);
            };
            float whole[4] = {};
            products(0, 0, whole);
            products(0, 2, small);
            if (all_parts) {
#pragma unroll
                for (int step = 0; step < 4; ++step)
#pragma unroll
                    for (int i = 0; i < 4; ++i) {
                        w[step][1][i] = round_pair(rest[step][i]);
                        w[step][2][i] = round_pair(minus_rounding(rest[step][i], w[step][1][i]));
                    }
                products(1, 1, small);
                products(2, 0, small);
            }
            products(0, 1, small);
            if (all_parts) products(1, 0, small);
#pragma unroll
            for (int i = 0; i < 4; ++i) sum[i] += whole[i];
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int r = 2 * quad + i % 2, of_tile = group + i / 2 * 8, col = tile * kFewTile + of_tile;
            if (r >= m) continue;
            float total = (sum[i] + small[i]) * low_of(kDown);
            if (!isfinite(total)) {
                const float *a = args.a + (size_t)r * args.lda, *w = args.w + (size_t)min(col, args.n - 1) * args.ldw;
                total = 0.0f;
#pragma unroll 1
                for (int k = k_begin; k < k_begin + columns; ++k) total = fmaf(a[k], w[k], total);
            }
            if (args.parts > 1) sums[r][warp * kFewTile + of_tile] = total;
            else if (col < args.n) args.c[(size_t)r * args.ldc + col] = total;
        }
    }
    asm volatile("cp.async.wait_group 0;" ::: "memory");
    if (args.parts > 1) {  // the first block of the cluster adds the parts in their order
        cg::this_cluster().sync();
        if (part == 0)
            for (int i = threadIdx.x; i < m * warps * kFewTile; i += threads) {
                const int r = i / (warps * kFewTile), c = i % (warps * kFewTile), col = block * warps * kFewTile + c;
                float v[4];
#pragma unroll
                for (int p = 0; p < 4; ++p)
                    if (p < args.parts) v[p] = cg::this_cluster().map_shared_rank(&sums[r][c], p)[0];
                float total = v[0];
#pragma unroll
                for (int p = 1; p < 4; ++p)
                    if (p < args.parts) total += v[p];
                if (col < args.n) args.c[(size_t)r * args.ldc + col] = total;
            }
        cluster_leave_together();
    }
}

template <int NB, int kRowsW, bool kEven>
static int launch(const CUtensorMap& map_a, const FloatArgs& args, cudaStream_t stream) {
    using P = Plan<NB, kRowsW>;
    auto kernel = gemm_f32_kernel<NB, kRowsW, kEven>;
    static DeviceSet devices{0};
    if (int status = reserve_shared("gemm_f32", kernel, P::kBytes, devices)) return status;
    const long long blocks = (long long)((args.n + kRowsW - 1) / kRowsW) * ((args.m + P::kRows - 1) / P::kRows) * args.parts;
    if (blocks > 0x7fffffff) return fail("gemm_f32: %d x %d results exceed the grid limit", args.m, args.n);
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3((unsigned)blocks);
    config.blockDim = dim3(kThreads);
    config.dynamicSmemBytes = P::kBytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = args.parts;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = dependent_launches_allowed() ? 2 : 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, kernel, map_a, args);
    if (status != cudaSuccess) return fail("gemm_f32: launch failed: %s", cudaGetErrorString(status));
    return check_launch("gemm_f32");
}

// How few rows are launched: a block to a multiprocessor, of the fewest warps that have a tile each, 16 that take tiles in turn where there
// are more.  (Two blocks of four warps, 3,072 x 2,048: 7.7 us, one of eight 8.0; 5,000 x 4,100: 26.5 and 25.4.)  Chunks under way: eight warps
// with two stages lose to the kernel of many rows (eight rows, 16,384 x 2,048: 38.4 us, and 33.3), which takes what finds no place here.
struct FewPlan {
    int warps, stages, bytes, blocks;
};
static FewPlan few_plan(const FloatArgs& args) {
    const long long rows = (long long)few_row(args.part_length / kChunk) * args.m * sizeof(uint2);
    const int tiles = (args.n + kFewTile - 1) / kFewTile;
    auto blocks = [&](int warps) { return (tiles + warps - 1) / warps * args.parts; };
    FewPlan plan{};
    for (int warps = blocks(4) <= 148 ? 4 : blocks(8) <= 148 ? 8 : 16; warps >= 4 && plan.warps == 0; warps = warps == 16 ? 8 : 0)
        for (int stages = warps == 16 ? 3 : 4; stages >= (warps == 16 ? 2 : 3) && plan.warps == 0; --stages) {
            const long long bytes = rows + stages * warps * kFewChunkBytes;
            if (bytes > kFewBytes) continue;
            plan.warps = warps, plan.stages = stages, plan.blocks = std::min(blocks(warps), 148);
            plan.bytes = (int)std::max<long long>(bytes, 116 * 1024);  // (so that there is no room for another block)
        }
    return plan;
}

template <bool kEven, int kStages>
static int launch_few(const FloatArgs& args, const FewPlan& plan, cudaStream_t stream) {
    auto kernel = gemm_f32_few_kernel<kEven, kStages>;
    static DeviceSet devices{0};
    if (int status = reserve_shared("gemm_f32", kernel, kFewBytes, devices)) return status;
    cudaLaunchConfig_t config = {};
    config.gridDim = dim3(plan.blocks);
    config.blockDim = dim3(32 * plan.warps);
    config.dynamicSmemBytes = plan.bytes;
    config.stream = stream;
    cudaLaunchAttribute attribute[2];
    attribute[0].id = cudaLaunchAttributeClusterDimension;
    attribute[0].val.clusterDim.x = args.parts;
    attribute[0].val.clusterDim.y = 1;
    attribute[0].val.clusterDim.z = 1;
    attribute[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attribute[1].val.programmaticStreamSerializationAllowed = 1;
    config.attrs = attribute;
    config.numAttrs = dependent_launches_allowed() ? 2 : 1;
    const cudaError_t status = cudaLaunchKernelEx(&config, kernel, args);
    if (status != cudaSuccess) return fail("gemm_f32: launch failed: %s", cudaGetErrorString(status));
    return check_launch("gemm_f32");
}

template <bool kEven>
static int launch_few_stages(const FloatArgs& args, const FewPlan& plan, cudaStream_t stream) {
    if (plan.stages == 4) return launch_few<kEven, 4>(args, plan, stream);
    return plan.stages == 3 ? launch_few<kEven, 3>(args, plan, stream) : launch_few<kEven, 2>(args, plan, stream);
}

template <int NB, int kRowsW>
static int launch_rows(const CUtensorMap& map_a, const FloatArgs& args, bool even, cudaStream_t stream) {
    return even ? launch<NB, kRowsW, true>(map_a, args, stream) : launch<NB, kRowsW, false>(map_a, args, stream);
}

static size_t plane_bytes(int m, int k) { return (size_t)m * ((k + kChunk - 1) / kChunk) * 128; }

}  // namespace mb

using namespace mb;

// Bytes of scratch that a product of m rows and k columns takes (0 for few rows); they start on a 16-byte boundary.
MB_EXPORT size_t mb_gemm_f32_scratch(int m, int k) {
    const int rows = std::min(m, kSlabRows);
    return m <= kInlineRows ? 0 : 3 * plane_bytes(rows, k);
}

// A: [m, k] with row stride lda; W: [n, k] with row stride ldw; C: [m, n] with row stride ldc.  `weights_ready` != 0 only for a W that no
// kernel still queued writes (a loaded weight): the kernels before start their followers early, and W is then read while they run.
MB_EXPORT int mb_gemm_f32(const float* a, int lda, const float* w, int ldw, float* c, int ldc, int m, int n, int k, void* scratch,
                          int weights_ready, cudaStream_t stream) {
    if (m <= 0 || n <= 0) return 0;
    if (k <= 0) return fail("gemm_f32: k %d must be positive", k);
    if (lda < k || ldw < k || ldc < n) return fail("gemm_f32: row strides (%d, %d, %d) are shorter than the rows (%d, %d, %d)", lda, ldw, ldc, k, k, n);
    if (m > kInlineRows && (scratch == nullptr || ((uintptr_t)scratch & 15))) return fail("gemm_f32: scratch for the split rows is missing or not on a 16-byte boundary");
    FloatArgs args{a, w, c, lda, ldw, ldc, m, n, k, 1, 0, weights_ready};
    // Parts of K, by n and k alone, so that every m gives a row the same bits: matrices of few tiles put more multiprocessors to work.
    const int tiles = (n + kTileN - 1) / kTileN;
    auto length = [&](int parts) { return ((k + parts - 1) / parts + kChunk - 1) / kChunk * kChunk; };
    args.parts = tiles <= 37 ? 4 : tiles <= 74 ? 2 : 1;
    while (args.parts > 1 && (k < 2 * kChunk * args.parts || length(args.parts) * (args.parts - 1) >= k)) args.parts /= 2;
    args.part_length = length(args.parts);
    const bool even_w = k % 4 == 0 && ldw % 4 == 0 && !((uintptr_t)w & 15), even_a = k % 4 == 0 && lda % 4 == 0 && !((uintptr_t)a & 15);
    if (m <= kFewRows) {
        const FewPlan plan = few_plan(args);
        if (plan.warps > 0) return even_w && even_a ? launch_few_stages<true>(args, plan, stream) : launch_few_stages<false>(args, plan, stream);
    }
    CUtensorMap map_a{};
    // More rows than 32 are split where they are multiplied, too, while tiles of 32 make no more blocks than multiprocessors: that saves the
    // kernel that splits (64 rows, 2,048 x 2,048: 14.4 -> 10.9 us, 2,048 x 8,192 38.4 -> 28.7, 301 rows, 256 x 64: 6.6 -> 2.7).  Element loads
    // stay with that kernel (64 rows, 2,048 x 8,192: 51 us, 90 with A inline).
    const long long blocks = (long long)tiles * args.parts * ((m + kInlineRows - 1) / kInlineRows);
    if (m <= kInlineRows || (blocks <= 148 && even_w && even_a)) {
        // 64 rows of W a block while that puts more multiprocessors to work.
        if (blocks <= 74) return launch_rows<1, 64>(map_a, args, even_w && even_a, stream);
        return launch_rows<1, 128>(map_a, args, even_w && even_a, stream);
    }
    const int chunks = (k + kChunk - 1) / kChunk;
    for (int first = 0; first < m; first += kSlabRows) {
        args.m = std::min(kSlabRows, m - first);
        args.a = a + (size_t)first * lda;
        args.c = c + (size_t)first * ldc;
        unsigned char* planes = static_cast<unsigned char*>(scratch);
        const unsigned blocks = (unsigned)(((size_t)args.m * chunks + 31) / 32);
        int status = even_a ? launch_dependent("gemm_f32", split_rows_kernel<true>, dim3(blocks), dim3(256), 0, stream, true, args.a, lda, args.m, k, chunks, planes)
                            : launch_dependent("gemm_f32", split_rows_kernel<false>, dim3(blocks), dim3(256), 0, stream, true, args.a, lda, args.m, k, chunks, planes);
        if (status) return status;
        // As few tiles of A as there must be, and these as low as that allows.
        const int a_tiles = (args.m + 159) / 160, rows = (args.m + a_tiles - 1) / a_tiles, nb = std::max(2, (rows + 31) / 32);
        if ((status = make_map(&map_a, planes, 3 * args.m, chunks * kChunk, chunks * kChunk, 32 * nb))) return status;
        switch (nb) {
            case 2: status = launch_rows<2, 128>(map_a, args, even_w, stream); break;
            case 3: status = launch_rows<3, 128>(map_a, args, even_w, stream); break;
            case 4: status = launch_rows<4, 128>(map_a, args, even_w, stream); break;
            default: status = launch_rows<5, 128>(map_a, args, even_w, stream);
        }
        if (status) return status;
    }
    return 0;
}

// 0 when no wait ever gave up; else 1 + (role << 8): 1 splitter, 2 and 3 issuer (operands, sums), 4 and 5 adder, 6 bringer.
MB_EXPORT int mb_gemm_f32_status() {
    int status = 0;
    if (cudaMemcpyFromSymbol(&status, g_gemm_status, sizeof(int)) != cudaSuccess) return -1;
    return status;
}
