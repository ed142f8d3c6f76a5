// Float32 values as three bfloat16 for products on the tensor cores: p1 + 2^-8 p2 + 2^-16 p3 (gemm_f32_tc.cu says
// which of the nine products of two such sums are taken, and how exact that is).  Parts two and three are kept
// multiplied by 2^8 and 2^16, at the first one's size: as they are, they would run into bfloat16's smallest number
// (2^-133) for values below 2^-110, of which 2e-7 was lost at 2^-112 and 1.5e-5 at 2^-118.  Like this every float32
// is its parts exactly, down to the smallest.  The instructions take the factors back out as they go from the small
// products to the large ones: the first of the next kind divides what the accumulator holds by 2^PART_SHIFT.
#pragma once
#include <stdint.h>

constexpr int PART_SHIFT = 8;

// Two neighbouring values as bfloat16 (lower half: the first), and what that leaves of them, times 2^PART_SHIFT.
__device__ __forceinline__ uint32_t bf16_part(float& x, float& y) {
    uint32_t two;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(two) : "f"(y), "f"(x));
    x = (x - __uint_as_float(two << 16)) * 256.f;
    y = (y - __uint_as_float(two & 0xffff0000u)) * 256.f;
    return two;
}
__device__ __forceinline__ bool finite(float v) { return fabsf(v) <= 3.402823466e38f; }
