// The float32 product's two ways: FFMA (gemm_f32.cu) and bfloat16 parts on the tensor cores (gemm_f32_tc.cu).
#pragma once
#include <cuda_runtime.h>

namespace mls_f32 {
constexpr int SKINNY_N = 256;        // up to so many columns the product is by rows, a warp a few outputs
// (gemm_f32.cu), unless they are 64 or more, as many values together as 64 of 4,096, and K is 2,048 (4,096 for float32
// rows, which are split first) or more.  us by rows / on tensor cores, bfloat16 rows, 64 x 4,096: 1 row 15.9 / 7.0, 64 rows
// 9.8 / 8.1, 512 15.9 / 11.8, 2,048 42.8 / 22.6; 128 x 2,048: 8.6 / 5.2, 7.4 / 6.3, 13.8 / 10.2, 49.3 / 19.2; float32 rows,
// 64 x 4,096: 15.2 / 8.4, 12.7 / 10.0, 15.5 / 16.1, 48.1 / 36.4, but 128 x 2,048, 256 rows 8.9 / 11.2.
constexpr int FEWEST_N = 64;
constexpr long long FEWEST_SIZE = 1 << 18;
// From so much of K on the tensor cores pay whatever M is (us after a flush of L2, FFMA / tensor cores: 1 x 300 x 2,048
// 18.5 / 14.1, 1 x 2,048 x 2,048 20.4 / 19.4, 9 x 2,048 x 2,048 82 / 19.5, 1 x 4,096 x 4,096 43 / 34, 16 x 4,096 x 4,096 162 / 36,
// 2,048 x 4,096 x 4,096 1,278 / 329; but 1 x 4,096 x 1,024 16.4 / 18.4), from a quarter of it
// where the weights are so many that their way from memory counts (1 x 16,384 x 1,024 39 / 32, 1 x 16,384 x 512
// 22.6 / 21.5; 1 x 8,192 x 1,024 is level, 22.5 / 23.6).
constexpr int TC_K = 2048;
constexpr long long TC_SIZE = 1 << 23;

// Whether the tensor cores take a product.  The types, N, K and the weights' address say so, never the rows: a row's
// bits do not depend on the rows it is computed with.
bool takes_tc(int a_dtype, const float* W, int N, int K);
long long tc_scratch_floats(const void* A, int a_dtype, int M, int N, int K);
int tc_launches(const void* A, int a_dtype, int M, int N, int K);
int product_tc(const void* A, int a_dtype, const float* W, float* out, int M, int N, int K, float* scratch,
               int* status, cudaStream_t stream);
}  // namespace mls_f32
