// The gated pairs of an epilogue that has many of them to a thread: the bits of gated_pair(), without its division.
#pragma once

#include "common.cuh"
#include "float_pairs.cuh"

namespace mb {

// x[i] / y[i] of two pairs, negated; y from 1 to 2^60, |x| up to 2^60.  The reciprocal's approximation (one unit of its last place) is corrected
// once, which rounds it to nearest, and so is the product with it, by the remainder, which an FMA has whole: this rounds to nearest
// (P. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, IBM J. Res. Dev. 34, 1990).  The signs are
// turned so that a zero keeps its own.
__device__ __forceinline__ uint64_t minus_quotients(uint64_t x, float y0, float y1) {
    float r0, r1;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r0) : "f"(-y0));
    asm("rcp.approx.f32 %0, %1;" : "=f"(r1) : "f"(-y1));
    const uint64_t y = pair_of(y0, y1);
    uint64_t r = pair_of(r0, r1);
    r = pair_fma(r, pair_fma(y, r, 0x3f8000003f800000ull), r);  // 1, 1
    const uint64_t q = pair_mul(x, r);
    return pair_fma(pair_fma(y, q, x), r, q);
}

__device__ __forceinline__ float min_of(float a, float b, float c) {  // NaN counts for nothing, as in fminf
    float m;
    asm("min.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}
__device__ __forceinline__ float max_of(float a, float b, float c) {
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(a), "f"(b), "f"(c));
    return m;
}

// z[i] <- 1 / (1 + e^(-z[i])), rounded as the division rounds it: with one number beyond e^40 by divisions, else side by side.
template <int kCount>
__device__ __forceinline__ void sigmoids(float (&z)[kCount]) {
    static_assert(kCount % 2 == 0, "whole pairs");
    float lowest = z[0];
#pragma unroll
    for (int i = 0; i < kCount; i += 2) lowest = min_of(lowest, z[i], z[i + 1]);
    if (lowest >= -40.0f) {
#pragma unroll
        for (int i = 0; i < kCount; i += 2) {
            const uint64_t q = minus_quotients(0x3f8000003f800000ull, 1.0f + expf(-z[i]), 1.0f + expf(-z[i + 1]));  // 1, 1
            z[i] = -low_of(q), z[i + 1] = -high_of(q);
        }
    } else {
#pragma unroll
        for (int i = 0; i < kCount; ++i) z[i] = 1.0f / (1.0f + expf(-z[i]));
    }
}

// gate[i] = gated_pair(activation, gate[i], up[i], clamp).  A division has a long way for unusual operands, and a branch to it after every pair
// keeps pairs from being worked on side by side; here one branch says whether all of a thread's gates are usual ones: exponentials up to e^40
// (every divisor then lies from 1 to 2^58, and no remainder that counts is below the floats), gates up to 2^60.  NaN passes through either way.
template <int kCount>
__device__ __forceinline__ void gate_pairs(int activation, float (&gate)[kCount], const float (&up)[kCount], const ClampedPair& clamp) {
    static_assert(kCount % 2 == 0, "whole pairs");
    if (activation == MB_ACT_SILU || activation == MB_ACT_CLAMPED_SWISH) {
        float lowest = gate[0], highest = gate[0];
#pragma unroll
        for (int i = 0; i < kCount; i += 2) lowest = min_of(lowest, gate[i], gate[i + 1]), highest = max_of(highest, gate[i], gate[i + 1]);
        if (activation == MB_ACT_SILU) {
            if (lowest >= -40.0f && highest <= 0x1p60f) {
#pragma unroll
                for (int i = 0; i < kCount; i += 2) {
                    const uint64_t q = minus_quotients(pair_of(gate[i], gate[i + 1]), 1.0f + expf(-gate[i]), 1.0f + expf(-gate[i + 1]));
                    gate[i] = -low_of(q) * up[i], gate[i + 1] = -high_of(q) * up[i + 1];
                }
                return;
            }
        } else if (clamp.slope >= 0x1p-30f && clamp.slope <= 0x1p30f && -clamp.slope * fminf(lowest, clamp.limit) <= 40.0f && fminf(highest, clamp.limit) <= 0x1p60f) {
#pragma unroll
            for (int i = 0; i < kCount; i += 2) {
                const float g0 = fminf(gate[i], clamp.limit), g1 = fminf(gate[i + 1], clamp.limit);
                const uint64_t q = minus_quotients(pair_of(g0, g1), 1.0f + expf(-clamp.slope * g0), 1.0f + expf(-clamp.slope * g1));
                gate[i] = -low_of(q) * (fminf(fmaxf(up[i], -clamp.limit), clamp.limit) + clamp.up_offset);
                gate[i + 1] = -high_of(q) * (fminf(fmaxf(up[i + 1], -clamp.limit), clamp.limit) + clamp.up_offset);
            }
            return;
        }
    }
#pragma unroll
    for (int i = 0; i < kCount; ++i) gate[i] = gated_pair(activation, gate[i], up[i], clamp);
}

}  // namespace mb
