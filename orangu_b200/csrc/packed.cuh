// Pairs of fp32 in one 64-bit register, every operation rounded by itself.
#pragma once

#include <stdint.h>

namespace ob {

namespace {

// The assembler fuses a packed product with the packed sum that follows it even when told not to (and takes a multiply-add by a
// literal 1 for a sum), so a sum is a multiply-add by a 1 that it cannot see: F2_ONES, handed to the kernel as an argument.
constexpr uint64_t F2_ONES = 0x3f8000003f800000ull;

__device__ __forceinline__ uint64_t f2_pack(uint32_t lo, uint32_t hi) {
    uint64_t v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(lo), "r"(hi));
    return v;
}
__device__ __forceinline__ uint64_t f2_pack(float lo, float hi) { return f2_pack(__float_as_uint(lo), __float_as_uint(hi)); }
__device__ __forceinline__ uint64_t f2_both(float v) { return f2_pack(v, v); }
__device__ __forceinline__ uint64_t f2_mul(uint64_t a, uint64_t b) {
    uint64_t v;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(v) : "l"(a), "l"(b));
    return v;
}
__device__ __forceinline__ uint64_t f2_add(uint64_t a, uint64_t b, uint64_t ones) {
    uint64_t v;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(v) : "l"(a), "l"(ones), "l"(b));
    return v;
}
__device__ __forceinline__ float f2_lo(uint64_t v) { return __uint_as_float((uint32_t)v); }
__device__ __forceinline__ float f2_hi(uint64_t v) { return __uint_as_float((uint32_t)(v >> 32)); }

}  // namespace

}  // namespace ob
