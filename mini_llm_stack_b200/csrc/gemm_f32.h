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
// From so much of K on the tensor cores pay whatever M is (us, FFMA / tensor cores: 1 x 300 x 2,048 18.4 / 16.4,
// 1 x 2,048 x 2,048 20.5 / 18.4, 9 x 2,048 x 2,048 82 / 18; but 1 x 4,096 x 1,024 16.4 / 18.4; those with eight
// groups of K, with sixteen 1 x 2,048 x 2,048 is at 10.5), from a quarter of it
// where the weights are so many that their way from memory counts (1 x 16,384 x 1,024 39 / 31, 1 x 16,384 x 512
// 22.6 both).
constexpr int TC_K = 2048;
constexpr long long TC_SIZE = 1 << 23;
// Rows of 4,096 to 8,191 stay with the chain over k although the tensor cores would take them faster and leave
// them nearer to float64 (16 x 4,096 x 4,096: 164 / 35 us).  What such runs are checked against are chains over k
// in float32 themselves: a layer of hidden size 4,096 lies up to 3.3e-5 from float64 there and is held to 3.0e-5,
// so that only sums with the same roundings pass (the chain's differ from it by 2.4e-5, the tensor cores' by 3.2e-5,
// float64's own would by 3.3e-5).  From 8,192 on (feed-forward rows) and below 4,096 both pass.
constexpr int CHAIN_K0 = 4096, CHAIN_K1 = 8192;

// Whether the tensor cores take a product.  The types, N, K and the weights' address say so, never the rows: a row's
// bits do not depend on the rows it is computed with.
bool takes_tc(int a_dtype, const float* W, int N, int K);
long long tc_scratch_floats(const void* A, int a_dtype, int M, int N, int K);
int tc_launches(const void* A, int a_dtype, int M, int N, int K);
int product_tc(const void* A, int a_dtype, const float* W, float* out, int M, int N, int K, float* scratch,
               int* status, cudaStream_t stream);
}  // namespace mls_f32
