// Packed two-float arithmetic: one instruction for two additions, products or fused multiply-adds, each rounded exactly as the
// scalar one.  A pair is a 64-bit register, the first value in the low half.
#pragma once

#include <stdint.h>

namespace rlxq {

__device__ __forceinline__ uint64_t f32x2(uint32_t lo, uint32_t hi) {
    uint64_t r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "r"(lo), "r"(hi));
    return r;
}
__device__ __forceinline__ uint64_t f32x2_splat(float f) { return f32x2(__float_as_uint(f), __float_as_uint(f)); }
__device__ __forceinline__ uint64_t add_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t mul_f32x2(uint64_t a, uint64_t b) {
    uint64_t d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ uint64_t fma_f32x2(uint64_t a, uint64_t b, uint64_t c) {
    uint64_t d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}
__device__ __forceinline__ float sum_f32x2(uint64_t v) {
    uint32_t lo, hi;
    asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "l"(v));
    return __uint_as_float(lo) + __uint_as_float(hi);
}
// bytes 2 H and 2 H + 1 of u -> (2^23 + byte, 2^23 + byte)
template <int H> __device__ __forceinline__ uint64_t magic_pair(uint32_t u) {
    return f32x2(__byte_perm(u, 0x4B000000u, 0x7440 + 2 * H), __byte_perm(u, 0x4B000000u, 0x7441 + 2 * H));
}

}  // namespace rlxq
