// Float32 values as sums of three bfloat16 for products on the tensor cores (gemm_f32_tc.cu says which of the
// nine products of two such sums are taken, and how exact that is).
//
// The third part of a value below 2^-110 runs into bfloat16's smallest number, 2^-133 (2e-7 of the value is lost at
// 2^-112, 1.5e-5 at 2^-118).  There are two ways around it:
//   - multiply by 2^16 first (gemm_f32_tc.cu): every float32, down to the smallest, is then its parts, but values from
//     2^112 on are infinite, which that product takes as chains of fmaf;
//   - keep the second and third part multiplied by 2^8 and 2^16 (bf16_part_up; the chunk-wise scans, whose order of
//     products suits it): the first product of the next larger kind divides what the accumulator holds by
//     2^PART_SHIFT.  No value is too large; float32's own denormal numbers keep fewer bits, for which the products left
//     out count.
#pragma once
#include <stdint.h>

// Two neighbouring float32 side by side (fma.rn.f32x2 and its like round each as a single one does).
__device__ __forceinline__ unsigned long long beside(uint32_t x, uint32_t y) {
    unsigned long long v;
    asm("mov.b64 %0, {%1, %2};" : "=l"(v) : "r"(x), "r"(y));
    return v;
}
__device__ __forceinline__ unsigned long long both_times(unsigned long long v, float f) {
    asm("mul.rn.f32x2 %0, %0, %1;" : "+l"(v) : "l"(beside(__float_as_uint(f), __float_as_uint(f))));
    return v;
}
// Two such values as bfloat16 (lower half: the first), and what that leaves of them.
__device__ __forceinline__ uint32_t bf16_part(unsigned long long& v) {
    float x, y;
    uint32_t two;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(two) : "f"(y), "f"(x));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(v) : "l"(beside(two << 16, two & 0xffff0000u)), "l"(0xbf800000bf800000ull));
    return two;
}
constexpr int PART_SHIFT = 8;
__device__ __forceinline__ uint32_t bf16_part_up(float& x, float& y) {
    unsigned long long v = beside(__float_as_uint(x), __float_as_uint(y));
    const uint32_t two = bf16_part(v);
    v = both_times(v, 256.f);
    asm("mov.b64 {%0, %1}, %2;" : "=f"(x), "=f"(y) : "l"(v));
    return two;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }
