// A float as three bfloat16 numbers that hold its 24 bits: its rounding, the rounding of what that left and of what this left.
#pragma once

#include "float_pairs.cuh"

#include <cuda_bf16.h>

namespace mb {

__device__ __forceinline__ uint32_t round_pair(uint64_t v) {
    const __nv_bfloat162 r = __floats2bfloat162_rn(low_of(v), high_of(v));
    return *reinterpret_cast<const uint32_t*>(&r);
}
__device__ __forceinline__ uint64_t minus_rounding(uint64_t v, uint32_t rounding) {
    return pair_fma(pair_of(__uint_as_float(rounding << 16), __uint_as_float(rounding & 0xffff0000u)), 0xbf800000bf800000ull, v);  // -1, -1
}
// Two floats as pairs of such numbers.
__device__ __forceinline__ void split_pair(uint64_t v, uint32_t& hi, uint32_t& mid, uint32_t& lo) {
    hi = round_pair(v);
    v = minus_rounding(v, hi);
    mid = round_pair(v);
    lo = round_pair(minus_rounding(v, mid));
}
__device__ __forceinline__ void split_pair(float a, float b, uint32_t& hi, uint32_t& mid, uint32_t& lo) { split_pair(pair_of(a, b), hi, mid, lo); }

// A sum that is finite only where eight floats are, and have three finite parts.  (The largest bfloat16 number is a little smaller than the
// largest float: four times what lies between them is infinite.)
__device__ __forceinline__ float fitness(const float (&x)[8]) {
    float sum = 0.0f;
#pragma unroll
    for (int j = 0; j < 8; ++j) sum = fmaf(x[j], 4.0f, sum);
    return sum;
}

}  // namespace mb
