// The chunk-wise form of the recurrences over a matrix state per head (chunk_scan.cu).
#pragma once
#include <cuda_runtime.h>

namespace mls_chunk {
constexpr int CHUNK = 64;            // tokens of a chunk

// Rows of an operand: element (t, head, i) lies at base[t * row + off + head * width + i].
struct Rows {
    const void* base;
    int dtype, row, off, width;
};

// How the state decays: one constant a head; a decay per token and key channel, the token read
// before it enters (with a bonus); mLSTM's gates with their stabiliser.
enum { HEAD_DECAY = 0, TOKEN_DECAY = 1, MLSTM = 2 };

struct Args {
    int mode;
    Rows q, k, v;
    int silu;                        // q, k and v pass through z * sigmoid(z) as they are read
    float q_scale;                   // MLSTM: what q is multiplied by
    const float* decay;              // HEAD_DECAY: [H]; TOKEN_DECAY: [T, H * e]
    const void* bonus;               // TOKEN_DECAY: [H * e] or null
    int bonus_dtype;
    // MLSTM
    const float* gates;              // [T, 2H]: input and forget pre-activations
    const void* bias_i;
    const void* bias_f;
    int bias_dtype;
    float cap;
    int n_groups;                    // copies of the stabiliser in a head's state
    float* den;                      // [T, H]

    const int* cu_q;
    const int* state_slot;
    float* state;
    long long slot_stride;           // floats between slots
    int head_stride;                 // floats between the heads of a slot
    int n_requests, n_heads, e, f;
    int least;                       // requests of at least so many tokens (>= 1); the others are left out
    float* out;                      // [T, H * f]
    int* status;                     // where a wait that runs out is noted
};

// Some of the chunks of a step, as many as scratch holds at a time: chunks [first, first + span) of `count`
// of the requests that go chunk by chunk, from the `from`th of them on; `chunks` in all.
struct Part {
    int from, count, first, span, chunks;
};

// Whether the chunk-wise kernels take these operands (alignment, sizes).
bool fits(const Args& a);
// Floats of scratch for so many chunks.
long long scratch_floats(int mode, int n_heads, int e, int f, long long chunks);
// The scan of a part.  A request's parts come one after the other, on one stream: each goes on from the
// state that the one before it left in the slot.
int scan(const Args& a, const Part& part, float* scratch, cudaStream_t stream);
}  // namespace mls_chunk
