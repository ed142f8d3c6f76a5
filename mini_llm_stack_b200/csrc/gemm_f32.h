// The float32 product's two ways: FFMA (gemm_f32.cu) and bfloat16 parts on the tensor cores (gemm_f32_tc.cu).
#pragma once
#include <cuda_runtime.h>

namespace mls_f32 {
constexpr int SKINNY_N = 256;        // up to so many columns the product is by rows, a warp a few outputs
// From so much of K on the tensor cores pay whatever M is (us, FFMA / tensor cores: 1 x 300 x 2,048 18.4 / 16.4,
// 1 x 2,048 x 2,048 20.5 / 18.4, 9 x 2,048 x 2,048 82 / 18; but 1 x 4,096 x 1,024 16.4 / 18.4), from a quarter of it
// where the weights are so many that their way from memory counts (1 x 16,384 x 1,024 39 / 31, 1 x 16,384 x 512
// 22.6 both).
constexpr int TC_K = 2048;
constexpr long long TC_SIZE = 1 << 23;

// Whether the tensor cores take a product.  N, K and the weights' address say so, never the rows: a row's
// bits do not depend on the rows it is computed with.
bool takes_tc(const float* W, int N, int K);
long long tc_scratch_floats(const void* A, int a_dtype, int M, int N, int K);
int product_tc(const void* A, int a_dtype, const float* W, float* out, int M, int N, int K, float* scratch,
               int* status, cudaStream_t stream);
}  // namespace mls_f32
