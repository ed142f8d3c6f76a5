// The gated delta rule's prepared rows, and its scan chunk by chunk (delta_chunk.cu).
#pragma once
#include <cuda_runtime.h>

namespace mls_delta {
// What the scan reads, float32, so that the tokens of a pass are one run of memory each:
//   [G][T][q: er | k: er]      [H][fr / 16][T][16 values]      [H][T][DR_SCALARS]
// with the scalars of a value head and token: decay, step, k . q, k' . k, k' . q, 0, 0, 0, where k'
// is the key of the token before (anything where a request's tokens of the step begin).
constexpr int DR_SCALARS = 8, DR_COLS = 16;
struct Prepared {
    size_t v_at, s_at;                 // where the values and the scalars begin
    size_t T;
    int er, fr;
    __host__ __device__ Prepared(int n_tokens, int H, int G, int er_, int fr_)
        : v_at((size_t)n_tokens * G * 2 * er_), s_at(v_at + (size_t)n_tokens * H * fr_),
          T((size_t)n_tokens), er(er_), fr(fr_) {}
    __host__ __device__ size_t qk(int kv, int t) const { return ((size_t)kv * T + t) * 2 * er; }
    __host__ __device__ size_t v(int head, int chunk, int t) const {
        return v_at + (((size_t)head * (fr / DR_COLS) + chunk) * T + t) * DR_COLS;
    }
    __host__ __device__ size_t scalars(int head, int t) const {
        return s_at + ((size_t)head * T + t) * DR_SCALARS;
    }
};
__host__ __device__ inline int prepared_floats(int H, int G, int er, int fr) {      // a token's share
    return 2 * G * er + H * (fr + DR_SCALARS);
}

// The tokens of requests of at least `least` tokens, chunk by chunk: of those requests `count` from the `from`th
// on, their chunks [first, first + span), `chunks` in all.
struct ChunkArgs {
    const float* rows;                 // as Prepared lays them out
    float* out;                        // [T, H f]
    float* state;
    long long state_stride;
    const int* cu_q;
    const int* state_slot;
    int n_tokens, n_requests, H, G, e, f, er, fr;
    int least, from, count, first, span, chunks;
    int* status;
    // the convolution's last inputs: columns of the projection, into the ring behind the state
    const float* proj;
    const int* positions;
    int width, qkv_col, taps, channels;
    long long ring_at;
};
bool chunk_fits(int er, int fr);
long long chunk_floats(int H, int G, int er);           // scratch of a chunk
int chunk_scan(const ChunkArgs& a, float* scratch, cudaStream_t stream);
}  // namespace mls_delta
