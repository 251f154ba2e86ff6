// Two floats side by side in a 64-bit register, as the paired float instructions take them.
#pragma once

#include <stdint.h>

namespace mb {

__device__ __forceinline__ uint64_t pair_of(float low, float high) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "f"(low), "f"(high));
    return v;
}
__device__ __forceinline__ uint64_t pair_fma(uint64_t a, uint64_t b, uint64_t c) {  // each rounded as fmaf rounds
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(b), "l"(c));
    return v;
}
__device__ __forceinline__ uint64_t pair_mul(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t pair_add(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ float low_of(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float high_of(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

}  // namespace mb
