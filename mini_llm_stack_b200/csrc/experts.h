// What the experts' two source files share.
#pragma once
#include "common.cuh"

namespace mls_experts {
// What a product does: the experts' down projection, or an up projection with a unit on its sums.
enum { DOWN = 0, GATED = 1, RELU2 = 2 };

constexpr int TC_EXPERTS = 4096;     // experts of a launch: their table lies beside the stages

// The gated unit on the two products' float32 sums.
__device__ __forceinline__ float gated_unit(float g, float u, float alpha, float limit) {
    if (limit > 0.f) {
        g = fminf(g, limit);
        u = fminf(fmaxf(u, -limit), limit);
        return times_sigmoid(g, alpha * g) * (u + 1.0f);
    }
    return times_sigmoid(g, g) * u;
}

// bfloat16 rows of whole 16-byte pieces at 16-byte addresses: the tensor cores'.
bool takes_tc(int dtype, const void* a, const void* w, int K);
// The product over sorted rows [n_slots, K], and the rows themselves.
int product_tc(int unit, const void* rows, const void* W, void* out, const int* order,
               const int* offsets, const float* weight, int scale, int n_slots, int n_experts, int N,
               int K, float alpha, float limit, int* status, cudaStream_t stream);
int gather_tc(const void* h, const int* order, const float* weight, int top, int scale, int n_slots,
              int K, void* rows, cudaStream_t stream);
}  // namespace mls_experts
