// Products of floats on the tensor cores (mma.sync m16n8k16) that keep a float's 24 bits: every operand is three bfloat16 numbers, its
// rounding, the rounding of what that left and of what this left, and six of the nine products of parts are added up in float (the
// other three are 2^-24 of the product at most: a second part is up to 2^-8 of its float, a third up to 2^-17).  Operands lie in shared
// memory as three planes, one after another.
#pragma once

#include "float_parts.cuh"

namespace mb {

using bf16 = __nv_bfloat16;
constexpr int kParts = 3;

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ldmatrix4(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void ldmatrix4_turned(uint32_t (&r)[4], uint32_t at) {
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(at) : "memory");
}
__device__ __forceinline__ void mma_bf16(float (&d)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};\n"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
// Two floats, and eight, into an operand's three planes.
__device__ __forceinline__ void split_two(float a, float b, bf16* at, int plane) {
    uint32_t hi, mid, lo;
    split_pair(a, b, hi, mid, lo);
    *reinterpret_cast<uint32_t*>(at) = hi;
    *reinterpret_cast<uint32_t*>(at + plane) = mid;
    *reinterpret_cast<uint32_t*>(at + 2 * plane) = lo;
}
__device__ __forceinline__ void store_parts(bf16* to, int plane, const float (&x)[8]) {
    uint4 hi, mid, lo;
    split_pair(x[0], x[1], hi.x, mid.x, lo.x);
    split_pair(x[2], x[3], hi.y, mid.y, lo.y);
    split_pair(x[4], x[5], hi.z, mid.z, lo.z);
    split_pair(x[6], x[7], hi.w, mid.w, lo.w);
    *reinterpret_cast<uint4*>(to) = hi;
    *reinterpret_cast<uint4*>(to + plane) = mid;
    *reinterpret_cast<uint4*>(to + 2 * plane) = lo;
}

// An array's elements moved up by kBy places: a loop that takes its elements one after another from the first places keeps one body and its
// array in registers.  Where a block runs a long loop's copies once each, all multiprocessors fetch their lines at the same time, about 100
// cycles for eight instructions: the chunks' solving kernel took 45 us with all of its loops unrolled, 36.5 with them rolled.
template <int kBy, typename T, int kCount>
__device__ __forceinline__ void move_up(T (&a)[kCount]) {
#pragma unroll
    for (int i = 0; i + kBy < kCount; ++i) a[i] = a[i + kBy];
}
template <int kBy, typename T, int kCount, int kInner>
__device__ __forceinline__ void move_up(T (&a)[kCount][kInner]) {
#pragma unroll
    for (int i = 0; i + kBy < kCount; ++i)
#pragma unroll
        for (int j = 0; j < kInner; ++j) a[i][j] = a[i + kBy][j];
}

using Parts = uint32_t[kParts][4];
__device__ __forceinline__ void load_parts(Parts& r, uint32_t at, int plane) {
#pragma unroll
    for (int i = 0; i < kParts; ++i) ldmatrix4(r[i], at + 2 * i * plane);
}
__device__ __forceinline__ void load_parts_turned(Parts& r, uint32_t at, int plane) {
#pragma unroll
    for (int i = 0; i < kParts; ++i) ldmatrix4_turned(r[i], at + 2 * i * plane);
}
// d[tile] += a . b for two neighbouring tiles of eight columns.  The tensor cores cut their sums off where a float addition rounds, so
// the sixteen products of roundings, whose sum has few bits to lose, and the smaller ones, the smallest first, start from zero and are
// added as floats (all in one chain: results of 2,048 tokens off by 8.9e-7 where the walk is off by 1e-7).
__device__ __forceinline__ void split_products(float (&d0)[4], float (&d1)[4], const Parts& a, const Parts& b) {
    float p0[4] = {}, p1[4] = {}, r0[4] = {}, r1[4] = {};
#pragma unroll
    for (int order = kParts - 1; order > 0; --order)
#pragma unroll
        for (int i = 0; i <= order; ++i) {
            mma_bf16(r0, a[i], b[order - i][0], b[order - i][1]);
            mma_bf16(r1, a[i], b[order - i][2], b[order - i][3]);
        }
    mma_bf16(p0, a[0], b[0][0], b[0][1]);
    mma_bf16(p1, a[0], b[0][2], b[0][3]);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {  // (two additions an instruction, each rounded as one by itself)
        const uint64_t s0 = pair_add(pair_of(d0[i], d0[i + 1]), pair_add(pair_of(p0[i], p0[i + 1]), pair_of(r0[i], r0[i + 1])));
        const uint64_t s1 = pair_add(pair_of(d1[i], d1[i + 1]), pair_add(pair_of(p1[i], p1[i + 1]), pair_of(r1[i], r1[i + 1])));
        d0[i] = low_of(s0), d0[i + 1] = high_of(s0), d1[i] = low_of(s1), d1[i + 1] = high_of(s1);
    }
}
// d = scale * d + a0 . b0 + a1 . b1 in the same way for one tile of eight columns and two steps of K; b: each part's two registers.
using HalfParts = uint32_t[kParts][2];
__device__ __forceinline__ void split_product_twice(float (&d)[4], float scale, const Parts& a0, const HalfParts& b0, const Parts& a1, const HalfParts& b1) {
    float p0[4] = {}, p1[4] = {}, r0[4] = {}, r1[4] = {};
#pragma unroll
    for (int order = kParts - 1; order > 0; --order)
#pragma unroll
        for (int i = 0; i <= order; ++i) {
            mma_bf16(r0, a0[i], b0[order - i][0], b0[order - i][1]);
            mma_bf16(r1, a1[i], b1[order - i][0], b1[order - i][1]);
        }
    mma_bf16(p0, a0[0], b0[0][0], b0[0][1]);
    mma_bf16(p1, a1[0], b1[0][0], b1[0][1]);
#pragma unroll
    for (int i = 0; i < 4; i += 2) {
        uint64_t sum = pair_fma(pair_of(d[i], d[i + 1]), pair_of(scale, scale), pair_add(pair_of(p0[i], p0[i + 1]), pair_of(r0[i], r0[i + 1])));
        sum = pair_add(sum, pair_add(pair_of(p1[i], p1[i + 1]), pair_of(r1[i], r1[i + 1])));
        d[i] = low_of(sum), d[i + 1] = high_of(sum);
    }
}

// A float from its parts, and the float dot product of two rows of parts.
__device__ __forceinline__ float whole_one(const bf16* at, int plane) {
    const float hi = __bfloat162float(at[0]);
    return isfinite(hi) ? hi + __bfloat162float(at[plane]) + __bfloat162float(at[2 * plane]) : hi;
}
template <int kCount>
__device__ __forceinline__ float whole_dot(const bf16* a, const bf16* b, int plane) {
    float sum = 0.0f;
#pragma unroll 1
    for (int i = 0; i < kCount; ++i) sum = fmaf(whole_one(a + i, plane), whole_one(b + i, plane), sum);
    return sum;
}
// acc += w . v token by token in float, for two tokens of a chunk a thread (`token` and 8 further on, its group's rows of the warp's 16) over
// the weights weight(token, earlier token) of the tokens up to each: what the tensor cores compute, but that a row of v that is not
// finite does not meet the zeros that stand for later tokens' weights.  `values`: the thread's pair of columns of the chunk's first row.
template <int kTiles, typename Weight>
__device__ __forceinline__ void causal_products(float (&acc)[kTiles][4], int token, Weight weight, const bf16* values, int row, int plane) {
    const int lane = threadIdx.x & 31, end = (token & ~15) + 16;
#pragma unroll 1
    for (int j0 = 0; j0 < end; j0 += 4) {  // a group's four lanes make a weight of either token each
        const int mine = j0 + (lane & 3);
        const float upper = mine <= token ? weight(token, mine) : 0.0f, lower = mine <= token + 8 ? weight(token + 8, mine) : 0.0f;
#pragma unroll 1
        for (int e = 0; e < 4; ++e) {
            const int j = j0 + e;
            const float first = __shfl_sync(0xffffffffu, upper, (lane & 28) + e), second = __shfl_sync(0xffffffffu, lower, (lane & 28) + e);
#pragma unroll
            for (int n = 0; n < kTiles; ++n) {
                const float x = whole_one(values + j * row + 8 * n, plane), y = whole_one(values + j * row + 8 * n + 1, plane);
                if (j <= token) acc[n][0] = fmaf(first, x, acc[n][0]), acc[n][1] = fmaf(first, y, acc[n][1]);
                if (j <= token + 8) acc[n][2] = fmaf(second, x, acc[n][2]), acc[n][3] = fmaf(second, y, acc[n][3]);
            }
        }
    }
}
// acc = S^T q for two tokens a thread, in float; `start`: the thread's pair of columns of the state's first row.
template <int kDim, int kTiles>
__device__ __forceinline__ void start_products(float (&acc)[kTiles][4], const bf16* queries, int query_row, int plane, const float* start, int columns) {
#pragma unroll
    for (int n = 0; n < kTiles; ++n) acc[n][0] = acc[n][1] = acc[n][2] = acc[n][3] = 0.0f;
#pragma unroll 1
    for (int d = 0; d < kDim; ++d) {
        const float first = whole_one(queries + d, plane), second = whole_one(queries + 8 * query_row + d, plane);
#pragma unroll
        for (int n = 0; n < kTiles; ++n) {
            const float2 s = *reinterpret_cast<const float2*>(start + (size_t)d * columns + 8 * n);
            acc[n][0] = fmaf(first, s.x, acc[n][0]), acc[n][1] = fmaf(first, s.y, acc[n][1]);
            acc[n][2] = fmaf(second, s.x, acc[n][2]), acc[n][3] = fmaf(second, s.y, acc[n][3]);
        }
    }
}

}  // namespace mb
