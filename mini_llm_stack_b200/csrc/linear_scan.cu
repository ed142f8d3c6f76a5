// Linear recurrences over a matrix state per head, carried from token to token in a
// float32 state slot per request, and what surrounds them.
//
// Per head, with key size e and value size f, the state S is [e, f] and one token does
//
//   read first  (a bonus u on the current token, a decay per key channel and token):
//       o_j = sum_i a_i (S_ij + u_i k_i v_j);   S_ij <- w_i S_ij + k_i v_j
//   write first (one fixed decay a head):
//       S_ij <- g S_ij + k_i v_j;               o_j = sum_i a_i S_ij
//
// with a the "receptance" or query.  mls_linear_scan walks the tokens of every request of
// the step in order, from the state the slot holds, and leaves o [T, H*f] in float32; the
// state goes back to the slot.  A CTA owns 16 columns of one head's S for one request:
// thread (column, row group) keeps every eighth row of its column in registers, a warp holds
// four columns times eight row groups, and the sum over i is the thread's rows in order
// followed by three shuffles: the order never depends on the batch or on how the tokens
// were cut into steps.  Tokens are taken 16 or 32 at a time through shared memory, four of
// them side by side where only the state's own update has to wait for the token before.
//
//   mls_scan_finish      o / rms(o) per head (eps inside the root) * weight * silu(gate)
//   mls_scan_finish_row  o / rms(o) over a token's whole row of heads * weight * sigmoid(gate)
//                        * a constant, into rows that may be wider than the heads
//   mls_rotate_rows      rotation of the first `dims` entries of every head of q and k,
//                        entry i paired with i + dims/2, k then times a constant; float32 out
//   mls_decay_lowrank    w = exp(-exp(W2 tanh(lo) + w0)) from the low-rank pre-activation
//                        (W2 handed over transposed)
//
// State, decays, exponentials, angles' cosines and sines, norms and sums are float32 (the
// angles themselves float64: position * frequency); a, k, v come from the projections, with
// `act` = 1 through silu (z * sigmoid(z), float32) as they are loaded.
#include "chunk_scan.h"
#include "common.cuh"
#include <limits.h>

namespace {
constexpr int LS_COLS = 16;         // columns of S a CTA owns
constexpr int LS_GROUPS = 8;        // row groups: lanes that share a column
constexpr int LS_THREADS = LS_COLS * LS_GROUPS;
constexpr int LS_UNROLL = 4;        // tokens whose sums over the row groups run side by side

// Four consecutive entries of a row as floats (the index a multiple of four, the row's start
// aligned to 16 bytes).
__device__ __forceinline__ float4 load4(const void* base, int dtype, size_t i) {
    if (dtype == MLS_BF16) {
        const uint2 raw = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)base + i);
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        return make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    return *reinterpret_cast<const float4*>((const float*)base + i);
}

__device__ __forceinline__ void store4(float* p, float4 v) { *reinterpret_cast<float4*>(p) = v; }
__device__ __forceinline__ void store4(__nv_bfloat16* p, float4 v) {
    *reinterpret_cast<uint2*>(p) = pack_bf16x4(v);
}

__device__ __forceinline__ float silu1(float z) { return times_sigmoid(z, z); }
__device__ __forceinline__ float4 silu4(float4 v) {
    return make_float4(silu1(v.x), silu1(v.y), silu1(v.z), silu1(v.w));
}

// (Four CTAs an SM up to 16 rows a thread: 592 places, so that the 512 CTAs of 32 heads with
// 256 value columns are one round and not two.)
template <int RPT, bool TOK_DECAY>
__global__ void __launch_bounds__(LS_THREADS, RPT <= 16 ? 4 : 2)
linear_scan_kernel(const void* __restrict__ a_src, int a_dtype, int a_row, int a_off,
                   const void* __restrict__ k_src, int k_dtype, int k_row, int k_off,
                   const void* __restrict__ v_src, int v_dtype, int v_row, int v_off,
                   const float* __restrict__ decay_tok, int decay_row,
                   const float* __restrict__ decay_head,
                   const void* __restrict__ bonus, int bonus_dtype, int read_first,
                   const int* __restrict__ cu_q, const int* __restrict__ state_slot,
                   float* __restrict__ state, long long state_stride,
                   int n_heads, int e, int f, int tokens_a_pass, float* __restrict__ out, int act,
                   int chunked_from) {
    chain_release();
    chain_wait();
    const int r = blockIdx.z, head = blockIdx.y, col0 = blockIdx.x * LS_COLS;
    const int t0 = cu_q[r], n = cu_q[r + 1] - t0;
    if (n <= 0 || n >= chunked_from) return;              // (longer requests: chunk_scan.cu's)
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int grp = lane & (LS_GROUPS - 1);               // row group: the low three lane bits
    const int my_col = warp * 4 + (lane >> 3);
    const int col = col0 + my_col;
    const bool col_ok = col < f;
    extern __shared__ float4 akw_s[];                     // [tokens][e]: (a, k, decay, -)
    float* v_s = reinterpret_cast<float*>(akw_s + (size_t)tokens_a_pass * e);   // [tokens][LS_COLS]

    float* S = state + (size_t)state_slot[r] * state_stride + (size_t)head * e * f;
    float s[RPT], ub[RPT];
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = i * LS_GROUPS + grp;
        s[i] = (col_ok && row < e) ? S[(size_t)row * f + col] : 0.f;
        ub[i] = (bonus && row < e) ? load_as_float(bonus, (size_t)head * e + row, bonus_dtype) : 0.f;
    }
    const float g = TOK_DECAY ? 1.f : decay_head[head];
    // whether every row of a, k, v and the decays can be read four entries at a time
    const bool vec4 = ((e | f | a_row | a_off | k_row | k_off | v_row | v_off) & 3) == 0 &&
                      (!TOK_DECAY || (decay_row & 3) == 0);
    float* out_col = out + (size_t)head * f + col;
    const size_t out_row = (size_t)n_heads * f;

    for (int b0 = 0; b0 < n; b0 += tokens_a_pass) {
        const int nb = min(tokens_a_pass, n - b0);
        __syncthreads();
        if (vec4) {
            // four consecutive entries a load, two such units a thread under way at a time
            const int e4 = e >> 2, units = nb * e4;
            for (int u0 = threadIdx.x; u0 < units; u0 += 2 * LS_THREADS) {
                float4 av[2], kv[2], wv[2];
                int at[2];
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int u = u0 + j * LS_THREADS;
                    at[j] = -1;
                    if (u < units) {
                        const int tt = u / e4, i = (u - tt * e4) << 2;
                        const size_t t = (size_t)(t0 + b0 + tt);
                        av[j] = load4(a_src, a_dtype, t * a_row + a_off + head * e + i);
                        kv[j] = load4(k_src, k_dtype, t * k_row + k_off + head * e + i);
                        if (act) {
                            av[j] = silu4(av[j]);
                            kv[j] = silu4(kv[j]);
                        }
                        wv[j] = TOK_DECAY ? *reinterpret_cast<const float4*>(
                                                decay_tok + t * decay_row + head * e + i)
                                          : make_float4(g, g, g, g);
                        at[j] = tt * e + i;
                    }
                }
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    if (at[j] >= 0) {
                        float4* dst = akw_s + at[j];
                        dst[0] = make_float4(av[j].x, kv[j].x, wv[j].x, 0.f);
                        dst[1] = make_float4(av[j].y, kv[j].y, wv[j].y, 0.f);
                        dst[2] = make_float4(av[j].z, kv[j].z, wv[j].z, 0.f);
                        dst[3] = make_float4(av[j].w, kv[j].w, wv[j].w, 0.f);
                    }
                }
            }
            for (int u = threadIdx.x; u < nb * (LS_COLS / 4); u += LS_THREADS) {
                const int tt = u / (LS_COLS / 4), j = (u - tt * (LS_COLS / 4)) << 2;
                const size_t t = (size_t)(t0 + b0 + tt);
                float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
                if (col0 + j < f)                      // f is a multiple of four here
                    x = load4(v_src, v_dtype, t * v_row + v_off + head * f + col0 + j);
                if (act) x = silu4(x);
                *reinterpret_cast<float4*>(v_s + tt * LS_COLS + j) = x;
            }
        } else {
            for (int u = threadIdx.x; u < nb * e; u += LS_THREADS) {
                const int tt = u / e, i = u - tt * e;
                const size_t t = (size_t)(t0 + b0 + tt);
                float4 x;
                x.x = load_as_float(a_src, t * a_row + a_off + head * e + i, a_dtype);
                x.y = load_as_float(k_src, t * k_row + k_off + head * e + i, k_dtype);
                x.z = TOK_DECAY ? decay_tok[t * decay_row + head * e + i] : g;
                x.w = 0.f;
                if (act) {
                    x.x = silu1(x.x);
                    x.y = silu1(x.y);
                }
                akw_s[u] = x;
            }
            for (int u = threadIdx.x; u < nb * LS_COLS; u += LS_THREADS) {
                const int tt = u / LS_COLS, j = u - tt * LS_COLS;
                const size_t t = (size_t)(t0 + b0 + tt);
                const float x = col0 + j < f
                    ? load_as_float(v_src, t * v_row + v_off + head * f + col0 + j, v_dtype) : 0.f;
                v_s[u] = act ? silu1(x) : x;
            }
        }
        __syncthreads();
        // LS_UNROLL tokens at a time: their sums over the row groups (three shuffles each)
        // run side by side, only the state's own chain is sequential
        for (int tt0 = 0; tt0 < nb; tt0 += LS_UNROLL) {
            float acc[LS_UNROLL];
#pragma unroll
            for (int u = 0; u < LS_UNROLL; ++u) {
                acc[u] = 0.f;
                const int tt = tt0 + u;
                if (tt < nb) {
                    const float vj = v_s[tt * LS_COLS + my_col];
                    const float4* row = akw_s + (size_t)tt * e + grp;
                    if (read_first) {
#pragma unroll
                        for (int i = 0; i < RPT; ++i) {
                            if (i * LS_GROUPS + grp < e) {
                                const float4 x = row[i * LS_GROUPS];
                                acc[u] = fmaf(x.x, fmaf(ub[i] * x.y, vj, s[i]), acc[u]);
                                s[i] = fmaf(x.z, s[i], x.y * vj);
                            }
                        }
                    } else {
#pragma unroll
                        for (int i = 0; i < RPT; ++i) {
                            if (i * LS_GROUPS + grp < e) {
                                const float4 x = row[i * LS_GROUPS];
                                s[i] = fmaf(x.z, s[i], x.y * vj);
                                acc[u] = fmaf(x.x, s[i], acc[u]);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int u = 0; u < LS_UNROLL; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], 1);
#pragma unroll
            for (int u = 0; u < LS_UNROLL; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], 2);
#pragma unroll
            for (int u = 0; u < LS_UNROLL; ++u) acc[u] += __shfl_xor_sync(0xffffffffu, acc[u], 4);
            if (grp == 0 && col_ok) {
#pragma unroll
                for (int u = 0; u < LS_UNROLL; ++u)
                    if (tt0 + u < nb) out_col[(size_t)(t0 + b0 + tt0 + u) * out_row] = acc[u];
            }
        }
    }
#pragma unroll
    for (int i = 0; i < RPT; ++i) {
        const int row = i * LS_GROUPS + grp;
        if (col_ok && row < e) S[(size_t)row * f + col] = s[i];
    }
}

// One warp a (token, head).  The gate's rows may be float32 whatever the output's type.
template <typename T>
__global__ void __launch_bounds__(128)
scan_finish_kernel(const float* __restrict__ o, const void* __restrict__ gate, int gate_dtype,
                   int gate_row, int gate_off, const void* __restrict__ w, int w_dtype, float eps,
                   T* __restrict__ out, int n_tokens, int n_heads, int f) {
    chain_release();
    chain_wait();
    const long long unit = (long long)blockIdx.x * 4 + (threadIdx.x >> 5);
    if (unit >= (long long)n_tokens * n_heads) return;
    const int lane = threadIdx.x & 31;
    const int t = (int)(unit / n_heads), head = (int)(unit % n_heads);
    const float* row = o + (size_t)t * n_heads * f + (size_t)head * f;
    float ss = 0.f;
    for (int j = lane; j < f; j += 32) ss = fmaf(row[j], row[j], ss);
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)f + eps);
    for (int j = lane; j < f; j += 32) {
        const int c = head * f + j;
        const float z = load_as_float(gate, (size_t)t * gate_row + gate_off + c, gate_dtype);
        float v = row[j] * inv;
        if (w) v *= load_as_float(w, c, w_dtype);
        Elem<T>::store(out + (size_t)t * n_heads * f + c, v * times_sigmoid(z, z));
    }
}

// The same for heads of up to 128 * QUADS values whose rows can be read four entries at a time: a
// lane keeps its quads in registers, and all loads are under way before the sum is taken.  (51 ->
// 30 us for 2,048 tokens of 32 heads of 256 values; 35 with the gate's type asked quad by quad.  Which of the two runs depends on the sizes
// alone.)
template <typename T, int QUADS>
__global__ void __launch_bounds__(256)
scan_finish_quads_kernel(const float* __restrict__ o, const void* __restrict__ gate, int gate_dtype,
                         int gate_row, int gate_off, const void* __restrict__ w, int w_dtype, float eps,
                         T* __restrict__ out, int n_tokens, int n_heads, int f) {
    chain_release();
    chain_wait();
    const long long unit = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (unit >= (long long)n_tokens * n_heads) return;
    const int lane = threadIdx.x & 31;
    const int t = (int)(unit / n_heads), head = (int)(unit % n_heads);
    const size_t at = (size_t)t * n_heads * f + (size_t)head * f;
    float4 v[QUADS], z[QUADS];
    float ss = 0.f;
    const size_t gate_at = (size_t)t * gate_row + gate_off + head * f;
    // (a load that is asked for inside a branch on its type is waited for there: one branch for all of them)
#pragma unroll
    for (int x = 0; x < QUADS; ++x)
        if (4 * (lane + 32 * x) < f) v[x] = *reinterpret_cast<const float4*>(o + at + 4 * (lane + 32 * x));
    if (QUADS == 1) {
        if (4 * lane < f) z[0] = load4(gate, gate_dtype, gate_at + 4 * lane);
    } else if (gate_dtype == MLS_BF16) {
        uint2 raw[QUADS];
#pragma unroll
        for (int x = 0; x < QUADS; ++x)
            if (4 * (lane + 32 * x) < f)
                raw[x] = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)gate + gate_at + 4 * (lane + 32 * x));
#pragma unroll
        for (int x = 0; x < QUADS; ++x) {
            const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[x].x));
            const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[x].y));
            z[x] = make_float4(lo.x, lo.y, hi.x, hi.y);
        }
    } else {
#pragma unroll
        for (int x = 0; x < QUADS; ++x)
            if (4 * (lane + 32 * x) < f)
                z[x] = *reinterpret_cast<const float4*>((const float*)gate + gate_at + 4 * (lane + 32 * x));
    }
#pragma unroll
    for (int x = 0; x < QUADS; ++x) {
        const int j = 4 * (lane + 32 * x);
        if (j >= f) continue;
        ss = fmaf(v[x].x, v[x].x, ss);
        ss = fmaf(v[x].y, v[x].y, ss);
        ss = fmaf(v[x].z, v[x].z, ss);
        ss = fmaf(v[x].w, v[x].w, ss);
    }
    const float inv = 1.0f / sqrtf(warp_sum(ss) / (float)f + eps);
#pragma unroll
    for (int x = 0; x < QUADS; ++x) {
        const int j = 4 * (lane + 32 * x);
        if (j >= f) continue;
        float4 n = make_float4(v[x].x * inv, v[x].y * inv, v[x].z * inv, v[x].w * inv);
        if (w) {
            const float4 m = load4(w, w_dtype, (size_t)head * f + j);
            n = make_float4(n.x * m.x, n.y * m.y, n.z * m.z, n.w * m.w);
        }
        const float4 g = silu4(z[x]);
        store4(out + at + j, make_float4(n.x * g.x, n.y * g.y, n.z * g.z, n.w * g.w));
    }
}

// One block a token: the norm runs over the token's whole row of heads.
template <typename T>
__global__ void __launch_bounds__(256)
scan_finish_row_kernel(const float* __restrict__ o, const T* __restrict__ gate, int gate_row,
                       int gate_off, const float* __restrict__ w, float eps, float out_scale,
                       T* __restrict__ out, long long out_row, int width) {
    chain_release();
    __shared__ float scratch[33];
    const int t = blockIdx.x;
    chain_wait();
    const float* row = o + (size_t)t * width;
    float ss = 0.f;
    for (int j = threadIdx.x; j < width; j += blockDim.x) ss = fmaf(row[j], row[j], ss);
    const float inv = 1.0f / sqrtf(block_sum(ss, scratch) / (float)width + eps);
    for (int j = threadIdx.x; j < width; j += blockDim.x) {
        const float z = Elem<T>::load(gate + (size_t)t * gate_row + gate_off + j);
        float v = row[j] * inv;
        if (w) v *= w[j];
        Elem<T>::store(out + (size_t)t * out_row + j, v * times_sigmoid(1.0f, z) * out_scale);
    }
}

// One block a token; thread (head, i) rotates the pair (i, i + dims/2) of q and of k.
template <typename T>
__global__ void __launch_bounds__(256)
rotate_rows_kernel(const T* __restrict__ src, int src_row, int q_off, int k_off,
                   const int* __restrict__ positions, const double* __restrict__ freq, int dims,
                   float k_scale, float* __restrict__ out, int n_heads, int e) {
    chain_release();
    extern __shared__ float cs[];                        // [dims]: cos | sin
    const int t = blockIdx.x, half = dims / 2;
    chain_wait();
    const int p = positions[t];
    for (int i = threadIdx.x; i < half; i += blockDim.x)
        angle_cos_sin(p, freq[i], cs[i], cs[half + i]);
    __syncthreads();
    const int width = n_heads * e;
    for (int u = threadIdx.x; u < 2 * width; u += blockDim.x) {
        const int which = u / width, c = u - which * width, i = c % e;
        const T* row = src + (size_t)t * src_row + (which ? k_off : q_off);
        float v = Elem<T>::load(row + c);
        if (i < dims) {
            const bool low = i < half;
            const float m = Elem<T>::load(row + (low ? c + half : c - half));
            const float co = cs[low ? i : i - half], si = cs[half + (low ? i : i - half)];
            v = low ? __fsub_rn(__fmul_rn(v, co), __fmul_rn(m, si))
                    : __fadd_rn(__fmul_rn(v, co), __fmul_rn(m, si));
        }
        out[(size_t)t * 2 * width + u] = which ? v * k_scale : v;
    }
}

// The same where pairs can be taken four at a time (half the rotated entries, heads and rows are
// whole quads): a thread takes a quad of first and the quad of second halves, or two quads that
// pass unchanged; the rows are on their way while the angles are worked out.  (62 -> 28 us for
// 2,048 tokens of 32 heads of 128; the same bits.)
constexpr int RQ_AT_ONCE = 4;
template <typename T>
__global__ void __launch_bounds__(256)
rotate_rows_quads_kernel(const T* __restrict__ src, int src_row, int q_off, int k_off,
                         const int* __restrict__ positions, const double* __restrict__ freq, int dims,
                         float k_scale, float* __restrict__ out, int n_heads, int e) {
    chain_release();
    extern __shared__ __align__(16) float cs[];          // [dims]: cos | sin
    const int t = blockIdx.x, half = dims / 2;
    chain_wait();
    const int width = n_heads * e, pairs = e / 8, units = 2 * n_heads * pairs;
    const int dt = sizeof(T) == 2 ? MLS_BF16 : MLS_F32;
    const T* row = src + (size_t)t * src_row;
    float* dst = out + (size_t)t * 2 * width;
    // unit: which of q and k, head, number of the pair of quads: those of the rotated halves first
    auto place = [&](int u, int& which, int& lo, int& hi, int& i) {
        which = u / (n_heads * pairs);
        const int x = u - which * n_heads * pairs, head = x / pairs, p = x - head * pairs;
        const bool turns = 4 * p < half;
        i = turns ? 4 * p : -1;
        const int first = turns ? 4 * p : dims + 8 * (p - half / 4);
        lo = head * e + first;
        hi = lo + (turns ? half : 4);
    };
    for (int u0 = threadIdx.x; u0 < units || u0 == (int)threadIdx.x; u0 += 256 * RQ_AT_ONCE) {
        float4 a[RQ_AT_ONCE], b[RQ_AT_ONCE];
#pragma unroll
        for (int x = 0; x < RQ_AT_ONCE; ++x) {
            const int u = u0 + 256 * x;
            if (u >= units) continue;
            int which, lo, hi, i;
            place(u, which, lo, hi, i);
            a[x] = load4(row + (which ? k_off : q_off), dt, lo);
            b[x] = load4(row + (which ? k_off : q_off), dt, hi);
        }
        if (u0 == (int)threadIdx.x) {                    // (once: every thread comes here first)
            const int p = positions[t];
            for (int i = threadIdx.x; i < half; i += blockDim.x)
                angle_cos_sin(p, freq[i], cs[i], cs[half + i]);
            __syncthreads();
        }
#pragma unroll
        for (int x = 0; x < RQ_AT_ONCE; ++x) {
            const int u = u0 + 256 * x;
            if (u >= units) continue;
            int which, lo, hi, i;
            place(u, which, lo, hi, i);
            float4 c = a[x], d = b[x];
            if (i >= 0)
                rotate_half4(a[x], b[x], *reinterpret_cast<const float4*>(cs + i),
                             *reinterpret_cast<const float4*>(cs + half + i), c, d);
            if (which) {
                c = make_float4(c.x * k_scale, c.y * k_scale, c.z * k_scale, c.w * k_scale);
                d = make_float4(d.x * k_scale, d.y * k_scale, d.z * k_scale, d.w * k_scale);
            }
            store4(dst + which * width + lo, c);
            store4(dst + which * width + hi, d);
        }
    }
}

// lo (float32 [T, rank], before its tanh) -> w [T, channels].  A block takes DL_TOKENS tokens
// and 256 channels: tanh(lo) of its tokens lies in shared memory, a thread owns one channel
// and reads its column of W2 (handed over transposed, [rank, channels], so that a warp reads
// consecutive floats) once for all its tokens.  k ascending: a token's sum does not depend
// on its block.
constexpr int DL_TOKENS = 16;
__global__ void __launch_bounds__(256)
decay_lowrank_kernel(const float* __restrict__ lo, int rank, const float* __restrict__ w2t,
                     const void* __restrict__ w0, int w0_dtype, float* __restrict__ out,
                     int n_tokens, int channels) {
    chain_release();
    extern __shared__ __align__(16) float th[];          // [DL_TOKENS][rank]
    const int t0 = blockIdx.y * DL_TOKENS, nt = min(DL_TOKENS, n_tokens - t0);
    const int c = blockIdx.x * 256 + threadIdx.x;
    chain_wait();
    for (int u = threadIdx.x; u < DL_TOKENS * rank; u += 256)
        th[u] = u < nt * rank ? tanhf(lo[(size_t)t0 * rank + u]) : 0.f;
    __syncthreads();
    if (c >= channels) return;
    float z[DL_TOKENS];
#pragma unroll
    for (int tt = 0; tt < DL_TOKENS; ++tt) z[tt] = 0.f;
    int i = 0;
    if ((rank & 3) == 0) {
        // four of the rank at a time: a 16-byte read of shared memory for four products (one a
        // product bounded the kernel: 34 -> 23 us for 1,501 tokens, rank 64, 2,048 channels)
#pragma unroll 2
        for (; i < rank; i += 4) {
            float w[4];
#pragma unroll
            for (int x = 0; x < 4; ++x) w[x] = w2t[(size_t)(i + x) * channels + c];
#pragma unroll
            for (int tt = 0; tt < DL_TOKENS; ++tt) {
                const float4 h = *reinterpret_cast<const float4*>(th + tt * rank + i);
                z[tt] = fmaf(w[0], h.x, z[tt]);
                z[tt] = fmaf(w[1], h.y, z[tt]);
                z[tt] = fmaf(w[2], h.z, z[tt]);
                z[tt] = fmaf(w[3], h.w, z[tt]);
            }
        }
    }
#pragma unroll 8
    for (; i < rank; ++i) {                              // (eight loads under way; the sums stay in order)
        const float w = w2t[(size_t)i * channels + c];
#pragma unroll
        for (int tt = 0; tt < DL_TOKENS; ++tt) z[tt] = fmaf(w, th[tt * rank + i], z[tt]);
    }
    const float b = load_as_float(w0, c, w0_dtype);
#pragma unroll
    for (int tt = 0; tt < DL_TOKENS; ++tt)
        if (tt < nt) out[(size_t)(t0 + tt) * channels + c] = expf(-expf(z[tt] + b));
}

template <int RPT>
int launch_scan(dim3 grid, size_t smem, cudaStream_t stream, const void* a_src, int a_dtype,
                int a_row, int a_off, const void* k_src, int k_dtype, int k_row, int k_off,
                const void* v_src, int v_dtype, int v_row, int v_off, const float* decay_tok,
                int decay_row, const float* decay_head, const void* bonus, int bonus_dtype,
                int read_first, const int* cu_q, const int* state_slot, float* state,
                long long state_stride, int n_heads, int e, int f, int tokens_a_pass, float* out,
                int act, int chunked_from) {
    auto kernel = decay_tok ? linear_scan_kernel<RPT, true> : linear_scan_kernel<RPT, false>;
    if (smem > 48 * 1024) {
        const int rc = (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem);
        if (rc) return rc;
    }
    MLS_LAUNCH(kernel, grid, dim3(LS_THREADS), smem, stream, a_src, a_dtype, a_row, a_off, k_src,
               k_dtype, k_row, k_off, v_src, v_dtype, v_row, v_off, decay_tok, decay_row,
               decay_head, bonus, bonus_dtype, read_first, cu_q, state_slot, state, state_stride,
               n_heads, e, f, tokens_a_pass, out, act, chunked_from);
    return launch_status();
}
}  // namespace

// `chunked_from`: requests of at least so many tokens are left out (mls_linear_scan_chunked takes
// them); 0: none.
MLS_API int mls_linear_scan(const void* a_src, int a_dtype, int a_row, int a_off,
                            const void* k_src, int k_dtype, int k_row, int k_off,
                            const void* v_src, int v_dtype, int v_row, int v_off,
                            const float* decay_tok, int decay_row, const float* decay_head,
                            const void* bonus, int bonus_dtype, int read_first, const int* cu_q,
                            const int* state_slot, float* state, long long state_stride,
                            int n_requests, int n_heads, int e, int f, float* out, int act,
                            int chunked_from, cudaStream_t stream) {
    if (n_requests <= 0) return 0;
    if (e <= 0 || f <= 0 || e > 32 * LS_GROUPS || (!decay_tok == !decay_head))
        return MLS_ERR_UNSUPPORTED;
    const dim3 grid((f + LS_COLS - 1) / LS_COLS, n_heads, n_requests);
    const int tokens_a_pass = e <= 64 ? 32 : 16;
    const size_t smem = (size_t)tokens_a_pass * (e * sizeof(float4) + LS_COLS * sizeof(float));
    const int rpt = (e + LS_GROUPS - 1) / LS_GROUPS;
#define LS_GO(R)                                                                                 \
    return launch_scan<R>(grid, smem, stream, a_src, a_dtype, a_row, a_off, k_src, k_dtype, k_row, \
                          k_off, v_src, v_dtype, v_row, v_off, decay_tok, decay_row, decay_head,  \
                          bonus, bonus_dtype, read_first, cu_q, state_slot, state, state_stride,  \
                          n_heads, e, f, tokens_a_pass, out, act,                                 \
                          chunked_from > 0 ? chunked_from : INT_MAX)
    if (rpt <= 2) LS_GO(2);
    if (rpt <= 4) LS_GO(4);
    if (rpt <= 8) LS_GO(8);
    if (rpt <= 16) LS_GO(16);
    LS_GO(32);
#undef LS_GO
}

// The same for prompts, chunk by chunk (chunk_scan.cu): a decay per token with the token read first,
// or one decay a head with the token taken in first and no bonus.  Of the requests of at least `least`
// tokens it takes `count` from the `from`th on: their chunks [first, first + span), `chunks` in all.
MLS_API int mls_linear_scan_chunked(const void* a_src, int a_dtype, int a_row, int a_off,
                                    const void* k_src, int k_dtype, int k_row, int k_off,
                                    const void* v_src, int v_dtype, int v_row, int v_off,
                                    const float* decay_tok, const float* decay_head,
                                    const void* bonus, int bonus_dtype, int read_first,
                                    const int* cu_q, const int* state_slot, float* state,
                                    long long state_stride, int n_requests, int n_heads,
                                    int e, int f, float* out, int act, int least,
                                    int from, int count, int first, int span, int chunks,
                                    float* scratch, int* status, cudaStream_t stream) {
    using namespace mls_chunk;
    if (n_requests <= 0) return 0;
    if (e <= 0 || f <= 0 || (!decay_tok == !decay_head) || (decay_tok && !read_first) ||
        (decay_head && (read_first || bonus)))
        return MLS_ERR_UNSUPPORTED;
    Args a{};
    a.mode = decay_tok ? TOKEN_DECAY : HEAD_DECAY;
    a.q = Rows{a_src, a_dtype, a_row, a_off, e};
    a.k = Rows{k_src, k_dtype, k_row, k_off, e};
    a.v = Rows{v_src, v_dtype, v_row, v_off, f};
    a.silu = act;
    a.decay = decay_tok ? decay_tok : decay_head;
    a.bonus = bonus;
    a.bonus_dtype = bonus_dtype;
    a.cu_q = cu_q;
    a.state_slot = state_slot;
    a.state = state;
    a.slot_stride = state_stride;
    a.head_stride = e * f;
    a.n_requests = n_requests;
    a.n_heads = n_heads;
    a.e = e;
    a.f = f;
    a.least = least;
    a.out = out;
    a.status = status;
    if (!fits(a)) return MLS_ERR_UNSUPPORTED;
    return scan(a, Part{from, count, first, span, chunks}, scratch, stream);
}

MLS_API int mls_scan_finish(const float* o, const void* gate, int gate_dtype, int gate_row,
                            int gate_off, const void* w, int w_dtype, float eps, void* out,
                            int act_dtype, int n_tokens, int n_heads, int f, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    const long long units = (long long)n_tokens * n_heads;
    const int blocks = (int)((units + 3) / 4);
    auto quads = [](const void* p, int dtype) {
        return reinterpret_cast<uintptr_t>(p) % (dtype == MLS_BF16 ? 8 : 16) == 0;
    };
    if (((f | gate_row | gate_off) & 3) == 0 && f <= 512 && quads(o, MLS_F32) && quads(gate, gate_dtype) &&
        quads(w, w_dtype) && quads(out, act_dtype)) {
#define QUADS_GO(T, N)                                                                             \
    MLS_LAUNCH((scan_finish_quads_kernel<T, N>), dim3((unsigned)((units + 7) / 8)), dim3(256), 0,  \
               stream, o, gate, gate_dtype, gate_row, gate_off, w, w_dtype, eps, (T*)out, n_tokens, \
               n_heads, f)
        if (act_dtype == MLS_BF16) {
            if (f <= 128) QUADS_GO(__nv_bfloat16, 1);
            else if (f <= 256) QUADS_GO(__nv_bfloat16, 2);
            else QUADS_GO(__nv_bfloat16, 4);
        } else {
            if (f <= 128) QUADS_GO(float, 1);
            else if (f <= 256) QUADS_GO(float, 2);
            else QUADS_GO(float, 4);
        }
#undef QUADS_GO
        return launch_status();
    }
    if (act_dtype == MLS_BF16)
        MLS_LAUNCH((scan_finish_kernel<__nv_bfloat16>), dim3(blocks), dim3(128), 0, stream, o,
                   gate, gate_dtype, gate_row, gate_off, w, w_dtype, eps,
                   (__nv_bfloat16*)out, n_tokens, n_heads, f);
    else
        MLS_LAUNCH((scan_finish_kernel<float>), dim3(blocks), dim3(128), 0, stream, o,
                   gate, gate_dtype, gate_row, gate_off, w, w_dtype, eps, (float*)out, n_tokens,
                   n_heads, f);
    return launch_status();
}

MLS_API int mls_scan_finish_row(const float* o, const void* gate, int act_dtype, int gate_row,
                                int gate_off, const float* w, float eps, float out_scale,
                                void* out, long long out_row, int n_tokens, int width,
                                cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (act_dtype == MLS_BF16)
        MLS_LAUNCH((scan_finish_row_kernel<__nv_bfloat16>), dim3(n_tokens), dim3(256), 0, stream, o,
                   (const __nv_bfloat16*)gate, gate_row, gate_off, w, eps, out_scale,
                   (__nv_bfloat16*)out, out_row, width);
    else
        MLS_LAUNCH((scan_finish_row_kernel<float>), dim3(n_tokens), dim3(256), 0, stream, o,
                   (const float*)gate, gate_row, gate_off, w, eps, out_scale, (float*)out, out_row,
                   width);
    return launch_status();
}

MLS_API int mls_rotate_rows(const void* src, int src_dtype, int src_row, int q_off, int k_off,
                            const int* positions, const double* freq, int dims, float k_scale,
                            float* out, int n_tokens, int n_heads, int e, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (dims < 0 || dims > e || (dims & 1) || (dims > 0 && !freq)) return MLS_ERR_UNSUPPORTED;
    const size_t smem = (size_t)(dims > 0 ? dims : 1) * sizeof(float);
    if (smem > 48 * 1024) return MLS_ERR_UNSUPPORTED;
    // (a block takes a token whatever its width: 2,048 rows of 128 entries take 6.9 us by quads and
    // 4.1 by pairs, of 256 6.9 and 5.5, of 512 7.2 and 8.7)
    if (n_heads * e >= 512 && e % 8 == 0 && dims % 8 == 0 && ((src_row | q_off | k_off) & 3) == 0 &&
        reinterpret_cast<uintptr_t>(src) % (src_dtype == MLS_BF16 ? 8 : 16) == 0 &&
        reinterpret_cast<uintptr_t>(out) % 16 == 0) {
        if (src_dtype == MLS_BF16)
            MLS_LAUNCH((rotate_rows_quads_kernel<__nv_bfloat16>), dim3(n_tokens), dim3(256), smem, stream,
                       (const __nv_bfloat16*)src, src_row, q_off, k_off, positions, freq, dims, k_scale,
                       out, n_heads, e);
        else
            MLS_LAUNCH((rotate_rows_quads_kernel<float>), dim3(n_tokens), dim3(256), smem, stream,
                       (const float*)src, src_row, q_off, k_off, positions, freq, dims, k_scale, out,
                       n_heads, e);
        return launch_status();
    }
    if (src_dtype == MLS_BF16)
        MLS_LAUNCH((rotate_rows_kernel<__nv_bfloat16>), dim3(n_tokens), dim3(256), smem, stream,
                   (const __nv_bfloat16*)src, src_row, q_off, k_off, positions, freq, dims,
                   k_scale, out, n_heads, e);
    else
        MLS_LAUNCH((rotate_rows_kernel<float>), dim3(n_tokens), dim3(256), smem, stream,
                   (const float*)src, src_row, q_off, k_off, positions, freq, dims, k_scale, out,
                   n_heads, e);
    return launch_status();
}

MLS_API int mls_decay_lowrank(const float* lo, int rank, const float* w2t, const void* w0,
                              int w0_dtype, float* out, int n_tokens, int channels,
                              cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    const size_t smem = (size_t)DL_TOKENS * rank * sizeof(float);
    if (rank <= 0 || smem > 48 * 1024) return MLS_ERR_UNSUPPORTED;
    const dim3 grid((channels + 255) / 256, (n_tokens + DL_TOKENS - 1) / DL_TOKENS);
    MLS_LAUNCH((decay_lowrank_kernel), grid, dim3(256), smem, stream, lo, rank, w2t, w0, w0_dtype,
               out, n_tokens, channels);
    return launch_status();
}
