// Recurrences over a matrix state per head, S <- decay S + k v^T, chunk by chunk for prompts.
//
// Token by token the state's chain of updates leaves most of an SM idle (0.16 to 0.9 us a token,
// whatever the arithmetic).  Within a chunk of 64 tokens that starts from state S0 the outputs are
//
//     o_t = (decay from the chunk's start to t) q_t S0 + sum_s P_ts v_s
//     P_ts = (decay from s to t) q_t . k_s           s <= t
//     S0'  = (the chunk's decay) S0 + sum_s (decay from s to the chunk's end) k_s v_s^T
//
// so that everything but the hand-over of states between chunks is matrix products, for all
// chunks, heads and requests at once:
//
//   scores   P of every chunk and head [64, 64]
//   update   U = sum_s (..) k_s v_s^T of every chunk and head [e, f]
//   carry    walks the chunks: leaves each chunk's S0 where its U was, and the last state in the slot
//   output   [q | P] x [S0; v], a product over e + 64
//
// All of it float32, on CUDA cores (fma.rn.f32x2) or, updates and outputs of wide heads, as bfloat16 parts on the
// tensor cores (chunk_scan_tc.cu).  Decays enter only as factors <= 1, never as the reciprocal of one.  Scores,
// the rows of q and k times their factors and each chunk's U are rounded to float32 once more than token by
// token; what a chunk saves is the state's own rounding a token.  Ops.CHUNKED_FROM says from where on that
// leaves outputs and states no further from float64.  Chunks are counted from a request's first token of the step.
//
// Measured (2,048 tokens, the scan's launches together, token by token -> all on CUDA cores -> now): retention of
// 32 heads of 128 x 256 1,825 -> 398 -> 225 us, mLSTM of 4 heads of 256 x 512 1,343 -> 238 -> 126; wkv of 32 heads of
// 64 x 64 581 -> 126 (its weights of pairs take a third of that).
//
// A token's value that is infinite or not a number reaches no earlier token: P is lower triangular, and a
// chunk with such a value multiplies its lower triangle only (0 x inf is not 0).  Requests never share a
// chunk.
//
// Bound by the states' way through memory (retention: U written, read and written by carry, read: 134 MB each, 82 us
// together), the loads that a block waits for before it multiplies, and where the products run on CUDA cores by
// the FFMA pipe: T H (2 e f + 64 (e + f)) multiply-adds.  Chunks of 64 balance the two: half the length doubles
// the states, twice the length doubles the products within chunks.
#include "chunk_common.cuh"

namespace {
using namespace mls_chunk;

typedef unsigned long long f32x2;
__device__ __forceinline__ f32x2 twice(float a) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %1};" : "=l"(r) : "f"(a));
    return r;
}
__device__ __forceinline__ void fma2(f32x2& c, f32x2 a, f32x2 b) {
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(a), "l"(b));
}
__device__ __forceinline__ float2 halves(f32x2 v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
// ------------------------------------------------------------------ tiles in shared memory
// 64 rows of K-contiguous values become T[k][row ^ 4 (k / 4 % 8)]: neither the stores (four rows,
// eight quads of k a warp) nor the reads of four rows at a time meet a bank twice.
__device__ __forceinline__ int turn(int k) { return 4 * ((k >> 2) & 7); }

// A thread's quads of such a tile: row and first of the four k of its y-th.
template <int THREADS>
constexpr int QUADS_OF = C * (C / 4) / THREADS;
template <int THREADS>
__device__ __forceinline__ int2 transposed_at(int y) {
    const int u = (threadIdx.x >> 5) + y * (THREADS / 32), lane = threadIdx.x & 31;
    return make_int2(4 * (u & 15) + (lane & 3), 4 * ((lane >> 2) + 8 * (u >> 4)));
}
__device__ __forceinline__ void put_transposed(float (*T)[C], int2 p, float4 v) {
    const int col = p.x ^ turn(p.y);
    T[p.y][col] = v.x;
    T[p.y + 1][col] = v.y;
    T[p.y + 2][col] = v.z;
    T[p.y + 3][col] = v.w;
}
// 64 rows (of k) of W values, as they are, from entry x0 of the operand's rows on; each(row, quad) as it goes by.
template <int THREADS, int W, typename Each>
__device__ __forceinline__ void fill_rows(float (*T)[W], const Reader& from, int x0, Each each) {
    constexpr int ALL = C * (W / 4) / THREADS, N = ALL < 8 ? ALL : 8;
    static_assert(ALL % N == 0, "whole batches");
#pragma unroll 1
    for (int y0 = 0; y0 < ALL; y0 += N) {
        float4 v[N];
        auto at = [&](int y) {
            const int u = threadIdx.x + (y0 + y) * THREADS;
            return make_int2(u / (W / 4), 4 * (u % (W / 4)));
        };
        from.quads<N>([&](int y) { const int2 p = at(y); return make_int2(p.x, x0 + p.y); }, v);
#pragma unroll
        for (int y = 0; y < N; ++y) {
            const int2 p = at(y);
            *reinterpret_cast<float4*>(&T[p.x][p.y]) = each(p.x, v[y]);
        }
    }
}

// acc += A x B over DEPTH of k, from k0: thread (ty, tx) owns rows 4 ty .. + 3 and 32 further on, columns
// 4 tx .. + 3 and, with eight columns a thread (TN), BN / 2 further on.  LOWER: row r of A ends at k = r,
// and what follows (zeros) is left out.
template <int BN, int TN, bool TURN_A, int DEPTH = C, bool LOWER = false>
__device__ __forceinline__ void multiply(f32x2 (&acc)[8][TN / 2], const float (*A)[C], const float (*B)[BN],
                                         int tx, int ty, int k0 = 0) {
#pragma unroll (LOWER ? 1 : 8)
    for (int k = k0; k < k0 + DEPTH; ++k) {
        const int ra = TURN_A ? (4 * ty) ^ turn(k) : 4 * ty;
        float v[8];
        *reinterpret_cast<float4*>(&v[0]) = *reinterpret_cast<const float4*>(&A[k][ra]);
        *reinterpret_cast<float4*>(&v[4]) = *reinterpret_cast<const float4*>(&A[k][ra + 32]);
        f32x2 b[TN / 2];
#pragma unroll
        for (int h = 0; h < TN / 4; ++h) {
            const ulonglong2 q = *reinterpret_cast<const ulonglong2*>(&B[k][4 * tx + h * (BN / 2)]);
            b[2 * h] = q.x;
            b[2 * h + 1] = q.y;
        }
#pragma unroll
        for (int i = 0; i < 8; ++i) {
            if (LOWER && 4 * ty + (i & 3) + 32 * (i >> 2) < k) continue;
            const f32x2 two = twice(v[i]);
#pragma unroll
            for (int j = 0; j < TN / 2; ++j) fma2(acc[i][j], two, b[j]);
        }
    }
}
// Every product adds up over runs of 16 of k, kept apart from the run being multiplied: chains of 16
// roundings and one a run.  With chains of 64 outputs had 1.2 times the token-by-token kernels' error at
// 130 tokens and states 1.02 times at 64; with runs of 16 both lie below it from Ops.CHUNKED_FROM on.
constexpr int SUMS = 16;
template <int N>
__device__ __forceinline__ void settle(f32x2 (&sum)[N], f32x2 (&acc)[N]) {
#pragma unroll
    for (int j = 0; j < N; ++j) {
        asm("add.rn.f32x2 %0, %0, %1;" : "+l"(sum[j]) : "l"(acc[j]));
        acc[j] = 0ull;
    }
}
template <int N>
__device__ __forceinline__ void clear(f32x2 (&acc)[8][N]) {
#pragma unroll
    for (int i = 0; i < 8; ++i)
#pragma unroll
        for (int j = 0; j < N; ++j) acc[i][j] = 0ull;
}

// ------------------------------------------------------------------------------- scores
// 4 x 4 scores a thread (the tile is small: warps count); the warps whose rows all lie before
// their columns have nothing to multiply.
template <int MODE>
__global__ void __launch_bounds__(256)
chunk_scores_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    __shared__ __align__(16) float A[C][C], B[C][C];
    __shared__ float power[C];
    __shared__ double la[C], lb[C];
    if (threadIdx.x < C) {
        if (MODE == HEAD_DECAY) power[threadIdx.x] = powf(a.decay[head], (float)threadIdx.x);
        if (MODE == MLSTM && threadIdx.x < w.n) {
            const double* lg = s.log_gates + ((w.idx * C + threadIdx.x) * a.n_heads + head) * 2;
            la[threadIdx.x] = lg[0];
            lb[threadIdx.x] = lg[1];
        }
    }
    const Reader q(a.q, a.silu, w, head), k(a.k, a.silu, w, head);
    // warps of 16 rows x 32 columns, threads of 4 x 4
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int r0 = (warp >> 1) * 16 + (lane >> 3) * 4, c0 = (warp & 1) * 32 + (lane & 7) * 4;
    const bool idle = (warp >> 1) * 16 + 15 < (warp & 1) * 32;
    f32x2 acc[4][2], sum[4][2];
#pragma unroll
    for (int i = 0; i < 4; ++i) acc[i][0] = acc[i][1] = sum[i][0] = sum[i][1] = 0ull;
    for (int i0 = 0; i0 < a.e; i0 += C) {
        __syncthreads();
        constexpr int N = QUADS_OF<256>;
        float4 x[N], y[N];
        auto place = [&](int g) { const int2 p = transposed_at<256>(g); return make_int2(p.x, i0 + p.y); };
        q.quads<N>(place, x);
        k.quads<N>(place, y);
#pragma unroll
        for (int g = 0; g < N; ++g) {
            put_transposed(A, transposed_at<256>(g), x[g]);
            put_transposed(B, transposed_at<256>(g), y[g]);
        }
        __syncthreads();
        if (idle) continue;
#pragma unroll 16
        for (int x = 0; x < C; ++x) {
            const float4 v = *reinterpret_cast<const float4*>(&A[x][r0 ^ turn(x)]);
            const ulonglong2 b = *reinterpret_cast<const ulonglong2*>(&B[x][c0 ^ turn(x)]);
            const float vs[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const f32x2 two = twice(vs[i]);
                fma2(acc[i][0], two, b.x);
                fma2(acc[i][1], two, b.y);
            }
            if (x % SUMS == SUMS - 1)
#pragma unroll
                for (int y = 0; y < 4; ++y) settle(sum[y], acc[y]);
        }
    }
    float* P = s.scores + (w.idx * a.n_heads + head) * C * C;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int t = r0 + i;
        const float2 lo = halves(sum[i][0]), hi = halves(sum[i][1]);
        float v[4] = {lo.x, lo.y, hi.x, hi.y};
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int j = c0 + x;
            if (j > t || t >= w.n) v[x] = 0.f;
            else if (MODE == HEAD_DECAY) v[x] *= power[t - j];
            else v[x] *= a.q_scale * expf((float)(la[t] + lb[j]));
        }
        *reinterpret_cast<float4*>(&P[t * C + c0]) = make_float4(v[0], v[1], v[2], v[3]);
    }
}

// A decay per token and channel.  The 64 tokens are four runs of 16, a run four steps of 4.  Inside
// a step the decays between two tokens are multiplied one by one; between steps of a run, and
// between runs, the weight of a pair is the product of the decays from its step's (run's) start
// to t, over whole steps (runs) between, and from s to its step's (run's) end, each at most 1: a
// thread takes a pair, no decay is ever divided by.
constexpr int RUN = 16, RUNS = C / RUN, STEP = 4, STEPS = C / STEP;
__device__ __forceinline__ float4 mul4(float4 x, float4 y) {
    return make_float4(x.x * y.x, x.y * y.y, x.z * y.z, x.w * y.w);
}
// Four products added up by themselves first: chains of e / 4 of them stay as exact as the
// token-by-token kernel's.
__device__ __forceinline__ float dot4(float4 x, float4 y, float v) {
    return v + fmaf(x.w, y.w, fmaf(x.z, y.z, fmaf(x.y, y.y, x.x * y.x)));
}
// Weights of four queries (from row t) and two keys (from row j) whose factors carry the decays up
// to the gap between them; `gap`: rows of decays between (gaps of them, e apart).
__device__ __forceinline__ void pairs_4x2(const float* r, const float* k, int pad, const float* gap, int gaps,
                                          int e, float (&v)[4][2]) {
#pragma unroll
    for (int x = 0; x < 4; ++x) v[x][0] = v[x][1] = 0.f;
#pragma unroll 2
    for (int i = 0; i < e; i += 4) {
        float4 y0 = *reinterpret_cast<const float4*>(k + i);
        float4 y1 = *reinterpret_cast<const float4*>(k + pad + i);
#pragma unroll
        for (int g = 0; g < 2; ++g)
            if (g < gaps) {
                const float4 d = *reinterpret_cast<const float4*>(gap + g * e + i);
                y0 = mul4(y0, d);
                y1 = mul4(y1, d);
            }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const float4 q = *reinterpret_cast<const float4*>(r + x * pad + i);
            v[x][0] = dot4(q, y0, v[x][0]);
            v[x][1] = dot4(q, y1, v[x][1]);
        }
    }
}

// QUADS: e / 4 where it is known (heads of 64), else 0.
template <int QUADS>
__global__ void __launch_bounds__(256)
chunk_scores_token_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    Where w;
    const int quads = QUADS ? QUADS : a.e / 4, e = 4 * quads, pad = e + 4;
    const int head = blockIdx.y;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    extern __shared__ __align__(16) float sm[];
    float* r_s = sm;                                     // [64][pad]
    float* k_s = r_s + C * pad;                          // [64][pad]
    float* w_s = k_s + C * pad;                          // [64][pad]
    float* step_s = w_s + C * pad;                       // [STEPS][e]: a step's decay
    float* run_s = step_s + STEPS * e;                   // [RUNS][e]: a run's
    float* bonus_s = run_s + RUNS * e;                   // [e]
    const int tid = threadIdx.x;
    const Reader q(a.q, a.silu, w, head), k(a.k, a.silu, w, head);
    float* P = s.scores + (w.idx * a.n_heads + head) * C * C;
    for (int u0 = tid; u0 < C * quads; u0 += 4 * 256) {
        float4 rq[4], rk[4], d[4];
        auto place = [&](int x) {                        // (past the last quad: a token past the chunk)
            const int u = u0 + 256 * x, t = u / quads;
            return make_int2(u < C * quads ? t : C, 4 * (u - t * quads));
        };
        q.quads<4>(place, rq);
        k.quads<4>(place, rk);
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int2 p = place(x);
            d[x] = make_float4(1.f, 1.f, 1.f, 1.f);
            if (p.x < w.n)
                d[x] = *reinterpret_cast<const float4*>(a.decay + ((size_t)(w.t0 + p.x) * a.n_heads + head) * e + p.y);
        }
#pragma unroll
        for (int x = 0; x < 4; ++x) {
            const int2 p = place(x);
            if (p.x >= C) continue;
            *reinterpret_cast<float4*>(r_s + p.x * pad + p.y) = rq[x];
            *reinterpret_cast<float4*>(k_s + p.x * pad + p.y) = rk[x];
            *reinterpret_cast<float4*>(w_s + p.x * pad + p.y) = d[x];
        }
    }
    for (int i = tid; i < e; i += 256)
        bonus_s[i] = a.bonus ? load_as_float(a.bonus, (size_t)head * e + i, a.bonus_dtype) : 0.f;
    for (int u = tid; u < C * C / 4; u += 256)           // keys of later steps
        if (u % (C / 4) > u / (C / 4) / STEP) reinterpret_cast<float4*>(P)[u] = make_float4(0.f, 0.f, 0.f, 0.f);
    __syncthreads();
    auto at4 = [&](const float* base, int t, int i) {
        return *reinterpret_cast<const float4*>(base + t * pad + i);
    };
    // inside the steps: thread (t, s of the same step)
    {
        const int t = tid >> 2, j = (t & ~3) + (tid & 3), gap = t - j - 1;
        float v = 0.f;
        if (j <= t) {
#pragma unroll 2
            for (int i = 0; i < e; i += 4) {
                float4 y = at4(k_s, j, i);
                if (j == t) y = mul4(y, *reinterpret_cast<const float4*>(bonus_s + i));
                if (gap > 0) y = mul4(y, at4(w_s, j + 1, i));
                if (gap > 1) y = mul4(y, at4(w_s, j + 2, i));
                v = dot4(at4(r_s, t, i), y, v);
            }
        }
        P[t * C + j] = v;
    }
    __syncthreads();
    // q from its step's start on, k up to its step's end
    for (int u = tid; u < STEPS * quads; u += 256) {
        const int g = u / quads, i = 4 * (u - g * quads), t = g * STEP;
        const float4 w0 = at4(w_s, t, i), w1 = at4(w_s, t + 1, i), w2 = at4(w_s, t + 2, i),
                     w3 = at4(w_s, t + 3, i);
        const float4 w01 = mul4(w0, w1), w23 = mul4(w2, w3);
        auto scale = [&](float* base, int x, float4 f) {
            float4* p = reinterpret_cast<float4*>(base + x * pad + i);
            *p = mul4(*p, f);
        };
        scale(r_s, t + 1, w0);
        scale(r_s, t + 2, w01);
        scale(r_s, t + 3, mul4(w01, w2));
        scale(k_s, t + 2, w3);
        scale(k_s, t + 1, w23);
        scale(k_s, t, mul4(w1, w23));
        *reinterpret_cast<float4*>(step_s + g * e + i) = mul4(w01, w23);
    }
    __syncthreads();
    // between the steps of a run: a thread takes a step's four queries and two keys before them
    if (tid < RUNS * 12) {
        const int run = tid / 12, x = tid % 12;          // steps 1, 2, 3 have 2, 4, 6 pairs of keys
        const int ga = x < 2 ? 1 : (x < 6 ? 2 : 3), pair = x - (ga == 1 ? 0 : (ga == 2 ? 2 : 6));
        const int t = run * RUN + ga * STEP, j = run * RUN + 2 * pair, gb = pair / 2;
        float v[4][2];
        pairs_4x2(r_s + t * pad, k_s + j * pad, pad, step_s + (run * (RUN / STEP) + gb + 1) * e,
                  ga - gb - 1, e, v);
#pragma unroll
        for (int y = 0; y < 4; ++y)
            *reinterpret_cast<float2*>(P + (t + y) * C + j) = make_float2(v[y][0], v[y][1]);
    }
    __syncthreads();
    // q from its run's start on, k up to its run's end
    for (int u = tid; u < C * quads; u += 256) {
        const int t = u / quads, i = 4 * (u - t * quads), g = t / STEP, g0 = g & ~(RUN / STEP - 1);
        float4 x = at4(r_s, t, i), y = at4(k_s, t, i);
#pragma unroll
        for (int h = 0; h < RUN / STEP; ++h) {
            const float4 d = *reinterpret_cast<const float4*>(step_s + (g0 + h) * e + i);
            if (g0 + h < g) x = mul4(x, d);
            if (g0 + h > g) y = mul4(y, d);
        }
        *reinterpret_cast<float4*>(r_s + t * pad + i) = x;
        *reinterpret_cast<float4*>(k_s + t * pad + i) = y;
    }
    for (int u = tid; u < RUNS * quads; u += 256) {
        const int g = u / quads, i = 4 * (u - g * quads);
        const float4* p = reinterpret_cast<const float4*>(step_s + g * (RUN / STEP) * e + i);
        *reinterpret_cast<float4*>(run_s + g * e + i) =
            mul4(mul4(p[0], p[quads]), mul4(p[2 * quads], p[3 * quads]));
    }
    __syncthreads();
    // between runs: a warp takes a pair of them (six), a thread four queries and two keys
    if (tid < 6 * 32) {
        const int x = tid >> 5, lane = tid & 31;
        const int ga = x == 0 ? 1 : (x < 3 ? 2 : 3), gb = x == 0 ? 0 : (x < 3 ? x - 1 : x - 3);
        const int t = ga * RUN + 4 * (lane >> 3), j = gb * RUN + 2 * (lane & 7);
        float v[4][2];
        pairs_4x2(r_s + t * pad, k_s + j * pad, pad, run_s + (gb + 1) * e, ga - gb - 1, e, v);
#pragma unroll
        for (int y = 0; y < 4; ++y)
            *reinterpret_cast<float2*>(P + (t + y) * C + j) = make_float2(v[y][0], v[y][1]);
    }
    // q from the chunk's start on, k up to the chunk's end, the whole chunk
#pragma unroll 2
    for (int u = tid; u < w.n * quads; u += 256) {
        const int t = u / quads, i = 4 * (u - t * quads), g = t / RUN;
        float4 x = at4(r_s, t, i), y = at4(k_s, t, i);
#pragma unroll
        for (int h = 0; h < RUNS; ++h) {
            const float4 d = *reinterpret_cast<const float4*>(run_s + h * e + i);
            if (h < g) x = mul4(x, d);
            if (h > g) y = mul4(y, d);
        }
        const size_t at = ((w.idx * C + t) * a.n_heads + head) * e + i;
        *reinterpret_cast<float4*>(s.rows_q + at) = x;
        *reinterpret_cast<float4*>(s.rows_k + at) = y;
    }
    for (int u = tid; u < quads; u += 256) {
        const float4* p = reinterpret_cast<const float4*>(run_s + 4 * u);
        *reinterpret_cast<float4*>(s.whole + (w.idx * a.n_heads + head) * e + 4 * u) =
            mul4(mul4(p[0], p[quads]), mul4(p[2 * quads], p[3 * quads]));
    }
}

// mLSTM's gates, a block a head and request, a warp a chunk, two neighbouring tokens a lane.  With F
// the sums of the log forget gates since the chunk's start (float64, so that differences of long
// sums lose nothing) the stabiliser m <- max(f + m, i) is F_t + max(m_0, max over s <= t of
// (i_s - F_s)): a chunk takes two scans over the lanes, and from chunk to chunk goes one number.
// What follows from it:
//   factor of q:  exp(F_t + m_0 - m_t) e^-1/2      factor of k:  exp(F_n - F_t + i_t - m_n)
//   of a pair:    exp((F_t - m_t) + (i_s - F_s))   of the state: exp(F_n + m_0 - m_n)
constexpr int GATE_WARPS = 16;
__global__ void __launch_bounds__(32 * GATE_WARPS)
chunk_gates_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    __shared__ double whole_s[GATE_WARPS], top_s[GATE_WARPS];
    __shared__ float m_s[GATE_WARPS + 1];
    const int head = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    Where w;
    if (!locate<true>(a, part, blockIdx.y, w)) return;
    float* m_slot = a.state + (size_t)a.state_slot[w.r] * a.slot_stride + (size_t)head * a.head_stride +
                    state_floats(MLSTM, a.e, a.f);
    const float bi = load_as_float(a.bias_i, head, a.bias_dtype),
                bf = load_as_float(a.bias_f, head, a.bias_dtype);
    const int t_end = a.cu_q[w.r + 1];
    if (threadIdx.x == 0) m_s[GATE_WARPS] = m_slot[0];
    for (int c0 = 0; c0 < w.chunks; c0 += GATE_WARPS) {
        const int c = c0 + warp, t0 = w.t0 + c * C, n = min(C, t_end - t0);
        double ig[2], F[2], top[2], earlier = -INFINITY;
        if (c < w.chunks) {
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                // past the chunk's end: nothing is forgotten, nothing enters
                const bool there = 2 * lane + x < n;
                const float* g = a.gates + (size_t)(t0 + min(2 * lane + x, n - 1)) * 2 * a.n_heads;
                const float z = a.cap * tanhf((g[a.n_heads + head] + bf) / a.cap);
                F[x] = there ? fminf(z, 0.f) - log1pf(expf(-fabsf(z))) : 0.f;
                ig[x] = there ? a.cap * tanhf((g[head] + bi) / a.cap) : -INFINITY;
            }
            F[1] += F[0];
            double sum = F[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double x = __shfl_up_sync(0xffffffffu, sum, o);
                if (lane >= o) sum += x;
            }
            F[0] += sum - F[1];
            F[1] = sum;
            top[0] = ig[0] - F[0];
            top[1] = fmax(top[0], ig[1] - F[1]);
            double most = top[1];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const double x = __shfl_up_sync(0xffffffffu, most, o);
                if (lane >= o) most = fmax(most, x);
            }
            const double before = __shfl_up_sync(0xffffffffu, most, 1);
            if (lane) earlier = before;
            if (lane == 31) {
                whole_s[warp] = F[1];
                top_s[warp] = most;
            }
        }
        __syncthreads();
        if (threadIdx.x == 0) {
            // m_s[x]: the stabiliser before the chunk of warp x; the last one: behind them all
            float m = m_s[GATE_WARPS];
            for (int x = 0; x < GATE_WARPS && c0 + x < w.chunks; ++x) {
                m_s[x] = m;
                m = (float)(whole_s[x] + fmax((double)m, top_s[x]));
                if (x + 1 < GATE_WARPS) m_s[x + 1] = m;
            }
            m_s[GATE_WARPS] = m;
        }
        __syncthreads();
        if (c < w.chunks) {
            const float m0 = m_s[warp];
            const float m_end = warp + 1 < GATE_WARPS ? m_s[warp + 1] : m_s[GATE_WARPS];
            const double whole = whole_s[warp];
#pragma unroll
            for (int x = 0; x < 2; ++x) {
                const int j = 2 * lane + x;
                if (j >= n) continue;
                const float m = (float)(F[x] + fmax((double)m0, fmax(earlier, top[x])));
                const size_t at = ((w.idx + c) * C + j) * a.n_heads + head;
                s.log_gates[2 * at] = F[x] - m;
                s.log_gates[2 * at + 1] = ig[x] - F[x];
                s.rows_q[at] = a.q_scale * expf((float)(F[x] + m0 - m));
                s.rows_k[at] = expf((float)(whole - F[x] + ig[x] - m_end));
                a.den[(size_t)(t0 + j) * a.n_heads + head] = expf(-m);   // the output kernel adds n . q to it
            }
            if (lane == 0) s.whole[(w.idx + c) * a.n_heads + head] = expf((float)(whole + m0 - m_end));
        }
        __syncthreads();
    }
    for (int g = threadIdx.x; g < a.n_groups; g += blockDim.x) m_slot[g] = m_s[GATE_WARPS];
}

// ------------------------------------------------------------------------------- update
// U[i, j] = sum_s factor_s k_s[i] v_s[j]; MLSTM: and n[i] = sum_s factor_s k_s[i].
// Tiles of 64 x 64, 8 x 4 a thread: the loads of a tile are hidden by the other blocks' arithmetic only,
// and more, smaller blocks hide them better (112 us against 116 at tiles of 64 x 128 for 2,048 tokens of
// 32 heads of 128 x 256; 16 against 28 for 1,501 tokens of 32 heads of 64 x 64).
template <int MODE>
__global__ void __launch_bounds__(128, 5)
chunk_update_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    constexpr int BN = C, TN = 4, THREADS = 128;
    __shared__ __align__(16) float A[C][C], B[C][BN];
    __shared__ float factor[C];
    const int f_tiles = (a.f + BN - 1) / BN;
    const int i0 = (blockIdx.x / f_tiles) * C, j0 = (blockIdx.x % f_tiles) * BN;
    if (threadIdx.x < C)
        factor[threadIdx.x] = row_factor<MODE>(a, s.rows_k, w, head, threadIdx.x, w.n - 1 - (int)threadIdx.x);
    __syncthreads();
    Rows kr = a.k;
    if (MODE == TOKEN_DECAY) kr = Rows{s.rows_k, MLS_F32, a.n_heads * a.e, 0, a.e};
    const Reader k(kr, MODE == TOKEN_DECAY ? 0 : a.silu, w, head, MODE == TOKEN_DECAY ? w.idx * C : (size_t)w.t0);
    const Reader v(a.v, a.silu, w, head);
    fill_rows<THREADS, C>(A, k, i0, [&](int t, float4 x) { return times(x, factor[t]); });
    fill_rows<THREADS, BN>(B, v, j0, [&](int, float4 x) { return x; });
    __syncthreads();
    const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
    f32x2 sum[8][TN / 2], acc[8][TN / 2];                  // (the factors are rounded already: short chains)
    clear(sum);
    clear(acc);
#pragma unroll 1
    for (int k0 = 0; k0 < C; k0 += SUMS) {
        multiply<BN, TN, false, SUMS>(acc, A, B, tx, ty, k0);
#pragma unroll
        for (int y = 0; y < 8; ++y) settle(sum[y], acc[y]);
    }
    float* U = s.states + (w.idx * a.n_heads + head) * state_floats(MODE, a.e, a.f);
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int i = i0 + 4 * ty + (x & 3) + 32 * (x >> 2);
        if (i >= a.e) continue;
#pragma unroll
        for (int h = 0; h < TN / 4; ++h) {
            const int j = j0 + 4 * tx + (BN / 2) * h;
            const float2 lo = halves(sum[x][2 * h]), hi = halves(sum[x][2 * h + 1]);
            if (j < a.f)
                *reinterpret_cast<float4*>(U + (size_t)i * a.f + j) = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    }
    if (MODE == MLSTM && j0 == 0 && threadIdx.x < C && i0 + threadIdx.x < a.e) {
        float n = 0.f;
#pragma unroll 16
        for (int t = 0; t < C; ++t) n += A[t][threadIdx.x];
        U[(size_t)a.e * a.f + i0 + threadIdx.x] = n;
    }
}

// -------------------------------------------------------------------------------- carry
// Four neighbouring entries of a head's state a thread, chunk after chunk; the loads of four
// chunks are under way together.
template <int MODE>
__global__ void __launch_bounds__(128)
chunk_carry_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<true>(a, part, blockIdx.z, w)) return;
    const int size = state_floats(MODE, a.e, a.f);
    const int at = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (at >= size) return;
    float4* slot = reinterpret_cast<float4*>(a.state + (size_t)a.state_slot[w.r] * a.slot_stride +
                                             (size_t)head * a.head_stride + at);
    const size_t step = (size_t)a.n_heads * size;
    float* U = s.states + (w.idx * a.n_heads + head) * size + at;
    const int len = a.cu_q[w.r + 1] - a.cu_q[w.r];
    const float g = MODE == HEAD_DECAY ? a.decay[head] : 0.f;
    const float g_whole = MODE == HEAD_DECAY ? powf(g, (float)C) : 0.f;
    float4 st = *slot;
    constexpr int AHEAD = 4;
    for (int c0 = 0; c0 < w.chunks; c0 += AHEAD) {
        float4 u[AHEAD];
        float d[AHEAD];
#pragma unroll
        for (int x = 0; x < AHEAD; ++x) {
            const int c = c0 + x;
            if (c >= w.chunks) continue;
            u[x] = *reinterpret_cast<const float4*>(U + c * step);
            if (MODE == HEAD_DECAY) {
                const int n = len - (w.c + c) * C;
                d[x] = n >= C ? g_whole : powf(g, (float)n);
            } else if (MODE == MLSTM) {
                d[x] = s.whole[(w.idx + c) * a.n_heads + head];
            } else {
                d[x] = s.whole[((w.idx + c) * a.n_heads + head) * a.e + at / a.f];   // f % 4 == 0
            }
        }
#pragma unroll
        for (int x = 0; x < AHEAD; ++x) {
            const int c = c0 + x;
            if (c >= w.chunks) continue;
            *reinterpret_cast<float4*>(U + c * step) = st;
            st = make_float4(fmaf(d[x], st.x, u[x].x), fmaf(d[x], st.y, u[x].y),
                             fmaf(d[x], st.z, u[x].z), fmaf(d[x], st.w, u[x].w));
        }
    }
    *slot = st;
}

// ------------------------------------------------------------------------------- output
// o = [P | factor q] x [v; S0]; MLSTM: and den_t = max(|[P | factor q] x [1; n]|, exp(-m_t)) + 1e-6.
// The first block of 64 is [P] x [v]; while a block is multiplied the next one's rows of S0 come by
// asynchronous copies and its rows of q into registers (without that, 2,048 tokens of 32 heads of
// 128 x 256: 200 us, now 166; 4 heads of 256 x 512: 113, now 85).
template <int MODE, int BN>
__global__ void __launch_bounds__(2 * BN, BN == 128 ? 2 : 3)
chunk_output_kernel(const Args a, const Scratch s, const Part part) {
    chain_release();
    chain_wait();
    Where w;
    const int head = blockIdx.y, j0 = blockIdx.x * BN;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    constexpr int THREADS = 2 * BN, TN = 4, QA = C * (C / 4) / THREADS;      // quads of A a thread brings in
    extern __shared__ __align__(16) float tiles[];
    float(*A)[C][C] = reinterpret_cast<float(*)[C][C]>(tiles);
    float(*B)[C][BN] = reinterpret_cast<float(*)[C][BN]>(tiles + 2 * C * C);
    __shared__ float factor[C], n_s[2][C];
    if (threadIdx.x < C)
        factor[threadIdx.x] = row_factor<MODE>(a, s.rows_q, w, head, threadIdx.x, threadIdx.x + 1);
    Rows qr = a.q;
    if (MODE == TOKEN_DECAY) qr = Rows{s.rows_q, MLS_F32, a.n_heads * a.e, 0, a.e};
    const Reader q(qr, MODE == TOKEN_DECAY ? 0 : a.silu, w, head, MODE == TOKEN_DECAY ? w.idx * C : (size_t)w.t0);
    const Reader v(a.v, a.silu, w, head);
    const size_t unit = w.idx * a.n_heads + head;
    const float* S = s.states + unit * state_floats(MODE, a.e, a.f);
    const float* P = s.scores + unit * C * C;
    const int tx = threadIdx.x % (BN / TN), ty = threadIdx.x / (BN / TN);
    const bool with_n = MODE == MLSTM && j0 == 0;
    const int blocks = 1 + (a.e + C - 1) / C;
    // rows i0 .. of S0 into buffer x (what is not there as zeros)
    auto ask_rows = [&](int i0, int x) {
#pragma unroll
        for (int u = threadIdx.x; u < C * (BN / 4); u += THREADS) {
            const int i = u / (BN / 4), j = 4 * (u % (BN / 4));
            const bool there = i0 + i < a.e && j0 + j < a.f;
            const float* src = there ? S + (size_t)(i0 + i) * a.f + j0 + j : S;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                         ::"r"((uint32_t)__cvta_generic_to_shared(&B[x][i][j])), "l"(src), "r"(there ? 16 : 0)
                         : "memory");
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    float4 next[QA];
#pragma unroll
    for (int y = 0; y < QA; ++y) {
        const int2 p = transposed_at<THREADS>(y);
        next[y] = *reinterpret_cast<const float4*>(P + p.x * C + p.y);
    }
#pragma unroll
    for (int y = 0; y < QA; ++y) put_transposed(A[0], transposed_at<THREADS>(y), next[y]);
    bool odd = false;                                          // a value that is not a number, or infinite
    fill_rows<THREADS, BN>(B[0], v, j0, [&](int, float4 x) {
        odd |= !((x.x + x.y + x.z + x.w) * 0.f == 0.f);        // (a sum that overflows: no harm)
        return x;
    });
    if (with_n && threadIdx.x < C) n_s[0][threadIdx.x] = 1.f;
    f32x2 acc[8][TN / 2], sum[8][TN / 2];
    clear(acc);
    clear(sum);
    float nq[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // short chains: the sum may nearly vanish
    odd = __syncthreads_or(odd);
    for (int b = 0; b < blocks; ++b) {
        const int x = b & 1, i0 = b * C;                       // i0: first row of the next block's S0
        const bool more = b + 1 < blocks;
        float n_next = 0.f;
        if (more) {
            ask_rows(i0, x ^ 1);
            q.quads<QA>([&](int y) { const int2 p = transposed_at<THREADS>(y); return make_int2(p.x, i0 + p.y); }, next);
            if (with_n && threadIdx.x < C && i0 + (int)threadIdx.x < a.e)
                n_next = S[(size_t)a.e * a.f + i0 + threadIdx.x];
        }
#pragma unroll 1
        for (int k0 = 0; k0 < C; k0 += SUMS) {
            if (odd && b == 0) multiply<BN, TN, true, SUMS, true>(acc, A[0], B[0], tx, ty, k0);
            else multiply<BN, TN, true, SUMS>(acc, A[x], B[x], tx, ty, k0);
#pragma unroll
            for (int y = 0; y < 8; ++y) settle(sum[y], acc[y]);
        }
        if (with_n && threadIdx.x < C) {
#pragma unroll 8
            for (int y = 0; y < C; ++y) nq[y & 7] = fmaf(A[x][y][threadIdx.x ^ turn(y)], n_s[x][y], nq[y & 7]);
        }
        if (more) {
#pragma unroll
            for (int y = 0; y < QA; ++y) {
                const int2 p = transposed_at<THREADS>(y);
                put_transposed(A[x ^ 1], p, times(next[y], factor[p.x]));
            }
            if (with_n && threadIdx.x < C) n_s[x ^ 1][threadIdx.x] = n_next;
        }
        asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        __syncthreads();
    }
    if (with_n && threadIdx.x < w.n) {
        float* den = a.den + (size_t)(w.t0 + threadIdx.x) * a.n_heads + head;
        const float all = ((nq[0] + nq[4]) + (nq[2] + nq[6])) + ((nq[1] + nq[5]) + (nq[3] + nq[7]));
        *den = fmaxf(fabsf(all), *den) + 1e-6f;
    }
    const int j = j0 + 4 * tx;
#pragma unroll
    for (int x = 0; x < 8; ++x) {
        const int t = 4 * ty + (x & 3) + 32 * (x >> 2);
        if (t >= w.n || j >= a.f) continue;
        const float2 lo = halves(sum[x][0]), hi = halves(sum[x][1]);
        *reinterpret_cast<float4*>(a.out + ((size_t)(w.t0 + t) * a.n_heads + head) * a.f + j) =
            make_float4(lo.x, lo.y, hi.x, hi.y);
    }
}

template <int MODE>
int update(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    const dim3 grid(((a.e + C - 1) / C) * ((a.f + C - 1) / C), a.n_heads, part.chunks);
    MLS_LAUNCH((chunk_update_kernel<MODE>), grid, dim3(128), 0, stream, a, s, part);
    return launch_status();
}
template <int MODE, int BN>
int output(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    constexpr int smem = 2 * C * (C + BN) * (int)sizeof(float);
    static bool configured = false;
    if (!configured) {
        const int rc = (int)cudaFuncSetAttribute(chunk_output_kernel<MODE, BN>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (rc) return rc;
        configured = true;
    }
    const dim3 grid((a.f + BN - 1) / BN, a.n_heads, part.chunks);
    MLS_LAUNCH((chunk_output_kernel<MODE, BN>), grid, dim3(2 * BN), smem, stream, a, s, part);
    return launch_status();
}

// The tensor cores take heads whose columns fill the 128 rows of an instruction (32 heads of 64 x 64 fill half
// of them: 1,501 tokens' updates 16.4 us either way, outputs 32.8 against 32.6) and whose rows fit shared memory.
bool takes_tc(const Args& a) { return a.e >= 64 && a.e <= 256 && a.f >= 128; }

size_t token_smem(int e) {
    return (size_t)(3 * C * (e + 4) + (STEPS + RUNS + 1) * e) * sizeof(float);
}

template <int MODE>
int launch(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    if (MODE == TOKEN_DECAY) {
        const size_t smem = token_smem(a.e);
        auto kernel = a.e == 64 ? chunk_scores_token_kernel<16> : chunk_scores_token_kernel<0>;
        const int rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (rc) return rc;
        MLS_LAUNCH(kernel, dim3(1, a.n_heads, part.chunks), dim3(256), smem,
                   stream, a, s, part);
    } else {
        if (MODE == MLSTM)
            MLS_LAUNCH((chunk_gates_kernel), dim3(a.n_heads, part.count), dim3(32 * GATE_WARPS), 0,
                       stream, a, s, part);
        MLS_LAUNCH((chunk_scores_kernel<MODE>), dim3(1, a.n_heads, part.chunks), dim3(256), 0,
                   stream, a, s, part);
    }
    const bool tensor_cores = takes_tc(a);
    int rc = tensor_cores ? update_tc<MODE>(a, s, part, stream) : update<MODE>(a, s, part, stream);
    if (rc) return rc;
    const int quads = state_floats(MODE, a.e, a.f) / 4;
    MLS_LAUNCH((chunk_carry_kernel<MODE>), dim3((quads + 127) / 128, a.n_heads, part.count), dim3(128),
               0, stream, a, s, part);
    rc = launch_status();
    if (rc) return rc;
    if (tensor_cores) return output_tc<MODE>(a, s, part, stream);
    // (a width of 64 leaves half of a wider tile empty)
    return a.f <= C ? output<MODE, 64>(a, s, part, stream)
                    : output<MODE, 128>(a, s, part, stream);
}
}  // namespace

namespace mls_chunk {
bool fits(const Args& a) {
    auto rows_fit = [](const Rows& r) {
        const size_t bytes = r.dtype == MLS_BF16 ? 8 : 16;
        return ((r.row | r.off | r.width) & 3) == 0 && reinterpret_cast<uintptr_t>(r.base) % bytes == 0;
    };
    if (!rows_fit(a.q) || !rows_fit(a.k) || !rows_fit(a.v) || (a.slot_stride & 3) || (a.head_stride & 3) ||
        reinterpret_cast<uintptr_t>(a.state) % 16 || reinterpret_cast<uintptr_t>(a.out) % 16)
        return false;
    if (a.mode == TOKEN_DECAY && (a.e > 128 || reinterpret_cast<uintptr_t>(a.decay) % 16)) return false;
    return a.n_heads <= 65535;
}

// (the float64 logarithms first, then sizes that are multiples of four floats)
long long scratch_floats(int mode, int n_heads, int e, int f, long long chunks) {
    long long n = (long long)state_floats(mode, e, f) + C * C;               // a chunk and head
    if (mode == TOKEN_DECAY) n += 2LL * C * e + e;
    if (mode == MLSTM) n += 4 * C + 2 * C + 1;
    return chunks * n_heads * n;
}

int scan(const Args& a, const Part& part, float* scratch, cudaStream_t stream) {
    if (part.count <= 0 || part.span <= 0 || part.chunks <= 0) return 0;
    if (part.chunks > 65535 || part.count > 65535 || part.from < 0 || part.first < 0 || a.least < 1)
        return MLS_ERR_UNSUPPORTED;
    const size_t units = (size_t)part.chunks * a.n_heads, rows = units * C;
    Scratch s{};
    float* at = scratch;
    if (a.mode == MLSTM) {
        s.log_gates = reinterpret_cast<double*>(at);
        at += 4 * rows;
    }
    s.states = at;
    at += units * state_floats(a.mode, a.e, a.f);
    s.scores = at;
    at += units * C * C;
    if (a.mode != HEAD_DECAY) {
        const size_t per = a.mode == TOKEN_DECAY ? rows * a.e : rows;
        s.rows_q = at;
        s.rows_k = at + per;
        s.whole = at + 2 * per;
    }
    if (a.mode == HEAD_DECAY) return launch<HEAD_DECAY>(a, s, part, stream);
    if (a.mode == TOKEN_DECAY) return launch<TOKEN_DECAY>(a, s, part, stream);
    return launch<MLSTM>(a, s, part, stream);
}
}  // namespace mls_chunk

// Floats of scratch that so many chunks of a chunk-wise scan take.
MLS_API long long mls_chunk_scratch_floats(int mode, int n_heads, int e, int f, long long chunks) {
    return scratch_floats(mode, n_heads, e, f, chunks);
}
