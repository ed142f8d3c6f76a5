// Float32 values as sums of three bfloat16 for products on the tensor cores (gemm_f32_tc.cu says which of the
// nine products of two such sums are taken, and how exact that is).
#pragma once
#include <stdint.h>

// Two neighbouring values as bfloat16 (lower half: the first), and what that leaves of them.
__device__ __forceinline__ uint32_t bf16_part(float& x, float& y) {
    uint32_t two;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(two) : "f"(y), "f"(x));
    x -= __uint_as_float(two << 16);
    y -= __uint_as_float(two & 0xffff0000u);
    return two;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }
