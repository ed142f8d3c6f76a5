// What the chunk-wise scans' kernels on CUDA cores (chunk_scan.cu) and on tensor cores (chunk_scan_tc.cu) share:
// where a block's chunk lies, and how its rows are read.
#pragma once
#include "chunk_scan.h"
#include "common.cuh"

namespace mls_chunk {
constexpr int C = CHUNK;

__device__ __forceinline__ float silu1(float z) { return times_sigmoid(z, z); }
__device__ __forceinline__ float4 times(float4 v, float f) {
    return make_float4(v.x * f, v.y * f, v.z * f, v.w * f);
}

// Where a block's chunk lies.
struct Where {
    int r, c;                        // request, chunk of the request
    int t0, n;                       // first token, tokens
    int chunks;                      // the request's chunks of this part
    size_t idx;                      // place among the part's chunks
};

// Chunk z of the part's chunks, or (REQUEST) the first one of its request z.  A request's length alone
// says whether it goes chunk by chunk.  Every thread calls; false: none.
template <bool REQUEST>
__device__ __forceinline__ bool locate(const Args& a, const Part& p, int z, Where& w) {
    __shared__ int at_s[2];          // request, place of its first chunk
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        int taken = -p.from, before = 0;   // the part's requests and chunks before these 32
        if (lane == 0) at_s[0] = -1;
        __syncwarp();
        for (int r0 = 0; r0 < a.n_requests; r0 += 32) {
            const int r = r0 + lane;
            const int len = r < a.n_requests ? a.cu_q[r + 1] - a.cu_q[r] : 0;
            const bool in = len >= a.least;
            const unsigned all = __ballot_sync(0xffffffffu, in);
            const int k = taken + __popc(all & ((1u << lane) - 1u));
            const int count = in && k >= 0 && k < p.count ? min(max((len + C - 1) / C - p.first, 0), p.span) : 0;
            int sum = count;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += x;
            }
            const int start = before + sum - count;
            const bool here = REQUEST ? in && k == z : z >= start && z < start + count;
            if (here) {
                at_s[0] = r;
                at_s[1] = start;
            }
            if (__any_sync(0xffffffffu, here)) break;
            taken += __popc(all);
            before += __shfl_sync(0xffffffffu, sum, 31);
        }
    }
    __syncthreads();
    w.r = at_s[0];
    if (w.r < 0) return false;
    const int j = REQUEST ? 0 : z - at_s[1];
    w.c = p.first + j;
    const int t = a.cu_q[w.r], len = a.cu_q[w.r + 1] - t;
    w.chunks = min(max((len + C - 1) / C - p.first, 0), p.span);
    w.idx = (size_t)(at_s[1] + j);
    w.t0 = t + w.c * C;
    w.n = min(C, len - w.c * C);
    return j < w.chunks;
}

// Quads of an operand's rows (zeros past the chunk and past the head's size).
struct Reader {
    const void* base;
    size_t row, at;                  // elements between tokens; the head's first entry
    int dtype, silu, n, size;
    __device__ __forceinline__ Reader(const Rows& r, int silu_, const Where& w, int head)
        : Reader(r, silu_, w, head, (size_t)w.t0) {}
    __device__ __forceinline__ Reader(const Rows& r, int silu_, const Where& w, int head, size_t t0)
        : base(r.base), row(r.row), at(t0 * r.row + r.off + (size_t)head * r.width),
          dtype(r.dtype), silu(silu_), n(w.n), size(r.width) {}
    // N quads, the x-th at (token, entry) = place(x): the type is asked once, so that their loads are under way
    // together (a load that is asked for inside a branch on its type is waited for there).
    template <int N, typename Place>
    __device__ __forceinline__ void quads(Place place, float4 (&v)[N]) const {
        if (dtype == MLS_BF16) {
            uint2 raw[N];
#pragma unroll
            for (int x = 0; x < N; ++x) {
                const int2 p = place(x);
                raw[x] = p.x < n && p.y < size ? *reinterpret_cast<const uint2*>((const __nv_bfloat16*)base + at +
                                                                                 (size_t)p.x * row + p.y)
                                               : make_uint2(0u, 0u);
            }
#pragma unroll
            for (int x = 0; x < N; ++x) {
                const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[x].x));
                const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[x].y));
                v[x] = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        } else {
#pragma unroll
            for (int x = 0; x < N; ++x) {
                const int2 p = place(x);
                v[x] = p.x < n && p.y < size
                           ? *reinterpret_cast<const float4*>((const float*)base + at + (size_t)p.x * row + p.y)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (silu)
#pragma unroll
            for (int x = 0; x < N; ++x)
                v[x] = make_float4(silu1(v[x].x), silu1(v[x].y), silu1(v[x].z), silu1(v[x].w));
    }
};

// What scores and gates leave for the products: a factor of q and of k for every token and head
// (HEAD_DECAY works them out itself), and the chunk's decay.  All of it by chunks, so that its size does
// not depend on the step's other tokens.
struct Scratch {
    double* log_gates;               // MLSTM: [chunks, 64, H, 2]
    float* states;                   // [chunks, H, e f (+ e)]
    float* scores;                   // [chunks, H, 64, 64]
    float* rows_q;                   // TOKEN_DECAY: [chunks, 64, H e]; MLSTM: factors [chunks, 64, H]
    float* rows_k;
    float* whole;                    // TOKEN_DECAY: [chunks, H, e]; MLSTM: [chunks, H]
};
__host__ __device__ inline int state_floats(int mode, int e, int f) {
    return e * f + (mode == MLSTM ? e : 0);
}

// Factors of the tokens' rows of q and k in this chunk.
template <int MODE>
__device__ __forceinline__ float row_factor(const Args& a, const float* factors, const Where& w, int head,
                                            int t, int power) {
    if (t >= w.n) return 0.f;
    if (MODE == HEAD_DECAY) return powf(a.decay[head], (float)power);
    if (MODE == MLSTM) return factors[(w.idx * C + t) * a.n_heads + head];
    return 1.f;
}

template <int MODE>
int update_tc(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream);
template <int MODE>
int output_tc(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream);
}  // namespace mls_chunk
