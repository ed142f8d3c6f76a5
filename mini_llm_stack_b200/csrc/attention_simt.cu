// Causal grouped-query attention over the paged cache on CUDA cores, for any
// mix of prompt portions and single decoded tokens.  It serves the float32 path
// (everything in 32-bit) and checks the tensor-core kernels of the bfloat16 path.
//
// Reference math (train/model.py:55-70): S = (q . k) * scale in float32; key j is
// hidden from the query at absolute position p iff j > p (the bottom-right
// aligned causal mask with p = i + Sk - Sq); P = softmax(S); O = P . V in
// float32, rounded once.  q head h reads kv head h / G.  With a window w, keys
// j <= p - w are hidden too.  With a cap c > 0 the score becomes c * tanh(S / c) before
// the softmax.  With sinks (one learned number per q head) the softmax's denominator also
// holds exp(sink_h): a term without key or value, not scaled and not capped.  With slopes
// (one number per q head) the score loses slope_h * (p - j), the distance to the key, before
// the cap.  With keep_first > 0 a window does not hide the sequence's first keep_first keys.
// With chunks of c tokens (and no window) the query at position p sees its own chunk, keys
// floor(p / c) c .. p.
// A row of `out` may be wider than the heads (out_stride elements a token).  The paged walk follows the reference's decode
// kernel (kernels/paged_attention.py:34-88): page = table[r, j / block],
// offset = j % block, online softmax over chunks of keys.
//
// Keys are taken 32 at a time from an absolute
// multiple of 32, so the order of every sum depends only on the token's own
// position and window: the result is bit-for-bit the same however the tokens
// were cut into steps and whatever else is in the batch.
//
// attention_simt_kernel: one warp per (token, q head), keys and values straight from the pages.
// attention_simt_tile_kernel: 32 rows (tokens x the q heads of a kv head) share every 32 keys
// through shared memory, eight rows a warp, with each row's operations in the same order: the same
// bits.  It takes the requests of at least TILE_LEN tokens; a warp a row read every key once a
// row, a key's row a lane, which touches 32 lines a load: 470 us for 515 tokens in three requests
// of 32 / 8 heads of 64 in float32, 71 us now (90 with the keys loaded between two barriers, 81 with a branch a row around
// its shuffles).  Bound by the chain of a block's steps: 32 keys' scores, maxima, exponentials and sums behind every barrier.
#include "common.cuh"

namespace {
constexpr int WARPS = 4;
constexpr int MOST_HD = 1024;         // heads of up to 512 entries take a smaller instantiation
constexpr int TILE_LEN = 8;           // tokens of a request from which on the tile kernel takes it

// q . k over one key row, accumulated in the order i = 0 .. hd-1.
__device__ __forceinline__ float dot_row(const float* q, const float* k, int hd) {
    float dot = 0.f;
    if ((hd & 3) == 0) {
        for (int i = 0; i < hd; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(k + i);
            dot = fmaf(q[i], v.x, dot);
            dot = fmaf(q[i + 1], v.y, dot);
            dot = fmaf(q[i + 2], v.z, dot);
            dot = fmaf(q[i + 3], v.w, dot);
        }
    } else {
        for (int i = 0; i < hd; ++i) dot = fmaf(q[i], k[i], dot);
    }
    return dot;
}
__device__ __forceinline__ float dot_row(const float* q, const __nv_bfloat16* k, int hd) {
    float dot = 0.f;
    if ((hd & 7) == 0) {
        for (int i = 0; i < hd; i += 8) {
            const uint4 raw = *reinterpret_cast<const uint4*>(k + i);
            const __nv_bfloat162* h2 = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const float2 f = __bfloat1622float2(h2[e]);
                dot = fmaf(q[i + 2 * e], f.x, dot);
                dot = fmaf(q[i + 2 * e + 1], f.y, dot);
            }
        }
    } else {
        for (int i = 0; i < hd; ++i) dot = fmaf(q[i], __bfloat162float(k[i]), dot);
    }
    return dot;
}

// SHORT: requests of TILE_LEN tokens and more are left out (an instantiation of its own: asked for in every
// launch, five registers more left six blocks an SM of seven, 16 prompts of eight tokens and 32 heads of
// 128 15 -> 21 us).
template <typename T, int MAX_HD, bool SHORT>
__global__ void __launch_bounds__(WARPS * 32)
attention_simt_kernel(const T* __restrict__ qkv, T* __restrict__ out,
                      const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                      const int* __restrict__ block_table, int max_blocks,
                      const int* __restrict__ positions, const int* __restrict__ req_of_token,
                      int n_tokens, int n_heads, int n_kv, int hd, int block_size, float scale,
                      int window, float softcap, long long n_pages,
                      const float* __restrict__ sink, const float* __restrict__ slopes,
                      int keep_first, long long out_stride, int chunk, const int* __restrict__ cu_q) {
    chain_release();
    chain_wait();
    __shared__ float q_s[WARPS][MAX_HD];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * WARPS + warp;   // (token, head)
    if (unit >= (long long)n_tokens * n_heads) return;
    const int t = (int)(unit / n_heads), h = (int)(unit % n_heads);
    const int kvh = h / (n_heads / n_kv);
    const int r = req_of_token[t];
    if (SHORT && cu_q[r + 1] - cu_q[r] >= TILE_LEN) return;         // the tile kernel's
    const int p = positions[t];
    const int row_w = (n_heads + 2 * n_kv) * hd;

    const T* qp = qkv + (size_t)t * row_w + (size_t)h * hd;
    for (int i = lane; i < hd; i += 32) q_s[warp][i] = Elem<T>::load(qp + i);
    __syncwarp();

    const int j_lo = max(0, first_visible(p, window, chunk));
    const int* table = block_table + (size_t)r * max_blocks;
    const int nd = (hd + 31) / 32;

    float m = -INFINITY, l = 0.f;
    float acc[MAX_HD / 32];
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) acc[i] = 0.f;

    const int keep = j_lo > 0 ? min(keep_first, j_lo) : 0;   // kept keys the window would hide
    const float slope = slopes ? slopes[h] : 0.f;
    for (int j0 = keep > 0 ? 0 : (j_lo / 32) * 32; j0 <= p; j0 += 32) {
        if (j0 >= keep && j0 + 32 <= j_lo) {          // past the kept keys: on to the window
            j0 = (j_lo / 32) * 32 - 32;
            continue;
        }
        const int j = j0 + lane;
        const bool valid = (j >= j_lo || j < keep) && j <= p;
        float s = -INFINITY;
        if (valid) {
            const int page = table[j / block_size];
            const T* kr = k_pool + (((size_t)kvh * n_pages + page) * block_size + j % block_size) * hd;
            s = dot_row(q_s[warp], kr, hd) * scale;
            if (slopes) s -= slope * (float)(p - j);
            if (softcap > 0.f) s = softcap * tanhf(s / softcap);
        }
        const float m_new = fmaxf(m, warp_max(s));
        const float pj = valid ? expf(s - m_new) : 0.f;
        const float corr = expf(m - m_new);       // m = -inf on the first chunk: exp(-inf) = 0
        l = l * corr + warp_sum(pj);
#pragma unroll
        for (int i = 0; i < MAX_HD / 32; ++i) acc[i] *= corr;
        for (int jj = 0; jj < 32; ++jj) {
            const int key = j0 + jj;
            if ((key < j_lo && key >= keep) || key > p) continue;        // uniform across the warp
            const float pk = __shfl_sync(0xffffffffu, pj, jj);
            const int page = table[key / block_size];
            const T* vr = v_pool + (((size_t)kvh * n_pages + page) * block_size + key % block_size) * hd;
#pragma unroll
            for (int i = 0; i < MAX_HD / 32; ++i) {
                const int dd = lane + 32 * i;
                if (i < nd && dd < hd) acc[i] = fmaf(pk, Elem<T>::load(vr + dd), acc[i]);
            }
        }
        m = m_new;
    }
    T* op = out + (size_t)t * out_stride + (size_t)h * hd;
    if (sink) l += expf(sink[h] - m);         // every token sees itself: m is a number
    const float inv = 1.0f / l;
#pragma unroll
    for (int i = 0; i < MAX_HD / 32; ++i) {
        const int dd = lane + 32 * i;
        if (i < nd && dd < hd) Elem<T>::store(op + dd, acc[i] * inv);
    }
}

constexpr int TILE_WARPS = 4, TILE_R = 8, TILE_ROWS = TILE_WARPS * TILE_R, KEYS = 32;

// ASYNC (float32): the next 32 keys come by asynchronous copies while these are worked on, into buffers of their
// own (a block waited for them, and for the page numbers before them, twice in every 32 keys).
template <int HD, bool ASYNC>
struct TileSmem {
    static constexpr int KP = HD + 4;                // a lane a key: 16-byte reads that meet no bank twice
    static constexpr int BUF = KEYS * (KP + HD);     // keys, then values
    static constexpr int Q = (ASYNC ? 2 : 1) * BUF, P = Q + TILE_ROWS * HD;
    static constexpr int FLOATS = P + TILE_ROWS * KEYS;
};

// Four neighbouring entries as floats (hd is a multiple of four).
__device__ __forceinline__ float4 quad(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 quad(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}

template <typename T, int HD>
__global__ void __launch_bounds__(TILE_WARPS * 32)
attention_simt_tile_kernel(const T* __restrict__ qkv, T* __restrict__ out,
                           const T* __restrict__ k_pool, const T* __restrict__ v_pool,
                           const int* __restrict__ block_table, int max_blocks,
                           const int* __restrict__ positions, const int* __restrict__ req_of_token,
                           int n_tokens, int n_heads, int n_kv, int hd, int block_size, float scale,
                           int window, float softcap, long long n_pages,
                           const float* __restrict__ sink, const float* __restrict__ slopes,
                           int keep_first, long long out_stride, int chunk,
                           const int* __restrict__ cu_q, int heads_a_block, int head_blocks) {
    chain_release();
    chain_wait();
    constexpr bool ASYNC = sizeof(T) == 4;
    using L = TileSmem<HD, ASYNC>;
    constexpr int ND = HD / 32;
    extern __shared__ __align__(16) float sm[];
    float* K_s = sm;
    float* V_s = sm + KEYS * L::KP;
    float* Q_s = sm + L::Q;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, quads = hd / 4;
    float* P_s = sm + L::P + warp * TILE_R * KEYS;
    const int group = n_heads / n_kv;
    const int kvh = blockIdx.y / head_blocks, head0 = kvh * group + (blockIdx.y % head_blocks) * heads_a_block;
    const int heads = min(heads_a_block, (kvh + 1) * group - head0);
    const int tokens = TILE_ROWS / heads_a_block;
    const int t_lo = (gridDim.x - 1 - blockIdx.x) * tokens;          // the latest tokens see the most keys
    const int t_hi = min(t_lo + tokens, n_tokens);
    const int row_w = (n_heads + 2 * n_kv) * hd;

    // row x of the block: token t_lo + x / heads_a_block, head head0 + x % heads_a_block
    for (int u = threadIdx.x; u < TILE_ROWS * quads; u += TILE_WARPS * 32) {
        const int x = u / quads, i = 4 * (u - x * quads), t = t_lo + x / heads_a_block, h = x % heads_a_block;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (t < t_hi && h < heads) v = quad(qkv + (size_t)t * row_w + (size_t)(head0 + h) * hd + i);
        *reinterpret_cast<float4*>(Q_s + x * HD + i) = v;
    }
    for (int s0 = t_lo; s0 < t_hi;) {
        const int r = req_of_token[s0];
        const int s1 = min(t_hi, cu_q[r + 1]);                       // a request's tokens lie together
        if (cu_q[r + 1] - cu_q[r] < TILE_LEN) {
            s0 = s1;
            continue;
        }
        // this warp's rows of the request
        int p[TILE_R], lo[TILE_R], keep[TILE_R];
        float m[TILE_R], l[TILE_R], slope[TILE_R], acc[TILE_R][ND];
#pragma unroll
        for (int y = 0; y < TILE_R; ++y) {
            const int x = warp * TILE_R + y, t = t_lo + x / heads_a_block, h = x % heads_a_block;
            const bool mine = t >= s0 && t < s1 && h < heads;
            p[y] = mine ? positions[t] : -1;
            lo[y] = mine ? max(0, first_visible(p[y], window, chunk)) : 0;
            keep[y] = lo[y] > 0 ? min(keep_first, lo[y]) : 0;
            slope[y] = slopes && mine ? slopes[head0 + h] : 0.f;
            m[y] = -INFINITY;
            l[y] = 0.f;
#pragma unroll
            for (int i = 0; i < ND; ++i) acc[y][i] = 0.f;
        }
        const int p_last = positions[s1 - 1];
        const int lo_first = max(0, first_visible(positions[s0], window, chunk));
        const int keep_most = min(keep_first, max(0, first_visible(p_last, window, chunk)));
        const int* table = block_table + (size_t)r * max_blocks;
        // the 32 keys from j on, or where they lie between the kept keys and the window the window's first ones
        auto tile_at = [&](int j) { return j >= keep_most && j + KEYS <= lo_first ? (lo_first / KEYS) * KEYS : j; };
        // where this thread's quad u of the keys from j0 on lies in the pools; false: nowhere
        auto place = [&](int j0, int u, size_t& at) {
            const int x = u / quads, i = 4 * (u - x * quads), j = j0 + x;
            const int page = j <= p_last && (j >= lo_first || j < keep_most) ? table[j / block_size] : -1;
            at = (((size_t)kvh * n_pages + max(page, 0)) * block_size + j % block_size) * hd + i;
            return page >= 0;
        };
        auto ask = [&](int j0, int buf) {
#pragma unroll 4
            for (int u = threadIdx.x; u < KEYS * quads; u += TILE_WARPS * 32) {
                const int x = u / quads, i = 4 * (u - x * quads);
                size_t at;
                const bool there = place(j0, u, at);
                const uint32_t k = (uint32_t)__cvta_generic_to_shared(sm + buf * L::BUF + x * L::KP + i);
                const uint32_t v = (uint32_t)__cvta_generic_to_shared(sm + buf * L::BUF + KEYS * L::KP + x * HD + i);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                             ::"r"(k), "l"(k_pool + (there ? at : 0)), "r"(there ? 16 : 0) : "memory");
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                             ::"r"(v), "l"(v_pool + (there ? at : 0)), "r"(there ? 16 : 0) : "memory");
            }
            asm volatile("cp.async.commit_group;\n" ::: "memory");
        };
        int j0 = tile_at(keep_most > 0 ? 0 : (lo_first / KEYS) * KEYS), buf = 0;
        if (ASYNC) {
            __syncthreads();                                         // (another request's keys may still be read)
            if (j0 <= p_last) ask(j0, 0);
        }
        for (int j_next; j0 <= p_last; j0 = j_next, buf ^= 1) {
            j_next = tile_at(j0 + KEYS);
            if (ASYNC) {
                asm volatile("cp.async.wait_group 0;\n" ::: "memory");
                __syncthreads();                                     // these are there, those before are read
                if (j_next <= p_last) ask(j_next, buf ^ 1);
                K_s = sm + buf * L::BUF;
                V_s = K_s + KEYS * L::KP;
            } else {
                __syncthreads();
#pragma unroll 2
                for (int u = threadIdx.x; u < KEYS * quads; u += TILE_WARPS * 32) {
                    const int x = u / quads, i = 4 * (u - x * quads);
                    float4 kv = make_float4(0.f, 0.f, 0.f, 0.f), vv = kv;
                    size_t at;
                    if (place(j0, u, at)) {
                        kv = quad(k_pool + at);
                        vv = quad(v_pool + at);
                    }
                    *reinterpret_cast<float4*>(K_s + x * L::KP + i) = kv;
                    *reinterpret_cast<float4*>(V_s + x * HD + i) = vv;
                }
                __syncthreads();
            }
            // rows that see some of these keys, and whether all of the warp's rows see all of them
            bool on[TILE_R], any = false, every = true;
#pragma unroll
            for (int y = 0; y < TILE_R; ++y) {
                on[y] = j0 <= p[y] && !(j0 >= keep[y] && j0 + KEYS <= lo[y]);
                any |= on[y];
                every &= on[y] && j0 + KEYS - 1 <= p[y] && (j0 >= lo[y] || j0 + KEYS <= keep[y]);
            }
            if (!any) continue;
            float s[TILE_R];
#pragma unroll
            for (int y = 0; y < TILE_R; ++y) s[y] = 0.f;
            const float* qw = Q_s + warp * TILE_R * HD;
            const float* kl = K_s + lane * L::KP;
#pragma unroll 4
            for (int i = 0; i < hd; i += 4) {
                const float4 k4 = *reinterpret_cast<const float4*>(kl + i);
#pragma unroll
                for (int y = 0; y < TILE_R; ++y) {
                    const float4 q4 = *reinterpret_cast<const float4*>(qw + y * HD + i);
                    s[y] = fmaf(q4.x, k4.x, s[y]);
                    s[y] = fmaf(q4.y, k4.y, s[y]);
                    s[y] = fmaf(q4.z, k4.z, s[y]);
                    s[y] = fmaf(q4.w, k4.w, s[y]);
                }
            }
            // (row beside row, without a branch between them: their shuffles and exponentials overlap)
            const int j = j0 + lane;
            float top[TILE_R], sum[TILE_R];
            bool valid[TILE_R];
#pragma unroll
            for (int y = 0; y < TILE_R; ++y) {
                valid[y] = on[y] && (j >= lo[y] || j < keep[y]) && j <= p[y];
                float v = s[y] * scale;
                if (slopes) v -= slope[y] * (float)(p[y] - j);
                if (softcap > 0.f) v = softcap * tanhf(v / softcap);
                top[y] = s[y] = valid[y] ? v : -INFINITY;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int y = 0; y < TILE_R; ++y) top[y] = fmaxf(top[y], __shfl_xor_sync(0xffffffffu, top[y], o));
#pragma unroll
            for (int y = 0; y < TILE_R; ++y) {
                const float m_new = fmaxf(m[y], top[y]);
                sum[y] = valid[y] ? expf(s[y] - m_new) : 0.f;
                P_s[y * KEYS + lane] = sum[y];
                // (0 on a row's first keys; a row that sees none of these stays as it is)
                const float corr = on[y] ? expf(m[y] - m_new) : 1.f;
                top[y] = corr;
#pragma unroll
                for (int i = 0; i < ND; ++i) acc[y][i] *= corr;
                if (on[y]) m[y] = m_new;
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1)
#pragma unroll
                for (int y = 0; y < TILE_R; ++y) sum[y] += __shfl_xor_sync(0xffffffffu, sum[y], o);
#pragma unroll
            for (int y = 0; y < TILE_R; ++y) l[y] = fmaf(l[y], top[y], sum[y]);
            __syncwarp();
            if (every) {
#pragma unroll 2
                for (int jj = 0; jj < KEYS; jj += 4) {
                    float4 pk[TILE_R];
#pragma unroll
                    for (int y = 0; y < TILE_R; ++y)
                        pk[y] = *reinterpret_cast<const float4*>(P_s + y * KEYS + jj);
#pragma unroll
                    for (int x = 0; x < 4; ++x) {
#pragma unroll
                        for (int i = 0; i < ND; ++i) {
                            const float v = V_s[(jj + x) * HD + lane + 32 * i];
#pragma unroll
                            for (int y = 0; y < TILE_R; ++y)
                                acc[y][i] = fmaf(x == 0 ? pk[y].x : (x == 1 ? pk[y].y : (x == 2 ? pk[y].z : pk[y].w)),
                                                 v, acc[y][i]);
                        }
                    }
                }
            } else {
                // (a key that a row does not see is not multiplied by zero: its value may be no number)
                int from[TILE_R], past[TILE_R], kept[TILE_R];        // a row's keys: [0, kept) and [from, past)
#pragma unroll
                for (int y = 0; y < TILE_R; ++y) {
                    past[y] = on[y] ? p[y] - j0 + 1 : 0;
                    from[y] = lo[y] - j0;
                    kept[y] = on[y] ? min(keep[y] - j0, past[y]) : 0;
                }
#pragma unroll 2
                for (int jj = 0; jj < KEYS; ++jj) {
                    float v[ND];
#pragma unroll
                    for (int i = 0; i < ND; ++i) v[i] = V_s[jj * HD + lane + 32 * i];
#pragma unroll
                    for (int y = 0; y < TILE_R; ++y) {
                        const float pk = P_s[y * KEYS + jj];
                        if (jj < kept[y] || (jj >= from[y] && jj < past[y])) {
#pragma unroll
                            for (int i = 0; i < ND; ++i) acc[y][i] = fmaf(pk, v[i], acc[y][i]);
                        }
                    }
                }
            }
            __syncwarp();
        }
#pragma unroll
        for (int y = 0; y < TILE_R; ++y) {
            if (p[y] < 0) continue;
            const int x = warp * TILE_R + y, t = t_lo + x / heads_a_block, h = head0 + x % heads_a_block;
            if (sink) l[y] += expf(sink[h] - m[y]);
            const float inv = 1.0f / l[y];
            T* op = out + (size_t)t * out_stride + (size_t)h * hd;
#pragma unroll
            for (int i = 0; i < ND; ++i) {
                const int dd = lane + 32 * i;
                if (dd < hd) Elem<T>::store(op + dd, acc[y][i] * inv);
            }
        }
        s0 = s1;
    }
}

template <typename T, int HD>
int launch_tile(const void* qkv, void* out, const void* k_pool, const void* v_pool, const int* block_table,
                int max_blocks, const int* positions, const int* req_of_token, int n_tokens, int n_heads,
                int n_kv, int hd, int block_size, float scale, int window, float softcap,
                long long n_pages, const float* sink, const float* slopes, int keep_first,
                long long out_stride, int chunk, const int* cu_q, cudaStream_t stream) {
    constexpr int smem = TileSmem<HD, sizeof(T) == 4>::FLOATS * (int)sizeof(float);
    static bool configured = false;
    if (!configured) {
        const int rc = (int)cudaFuncSetAttribute(attention_simt_tile_kernel<T, HD>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (rc) return rc;
        configured = true;
    }
    const int group = n_heads / n_kv, heads = group < TILE_ROWS ? group : TILE_ROWS;
    const int head_blocks = (group + heads - 1) / heads, tokens = TILE_ROWS / heads;
    MLS_LAUNCH((attention_simt_tile_kernel<T, HD>), dim3((n_tokens + tokens - 1) / tokens, n_kv * head_blocks),
               dim3(TILE_WARPS * 32), smem, stream, (const T*)qkv, (T*)out, (const T*)k_pool,
               (const T*)v_pool, block_table, max_blocks, positions, req_of_token, n_tokens, n_heads, n_kv,
               hd, block_size, scale, window, softcap, n_pages, sink, slopes, keep_first, out_stride, chunk,
               cu_q, heads, head_blocks);
    return launch_status();
}
}  // namespace

MLS_API int mls_attention_simt(const void* qkv, void* out, int dtype, const void* k_pool,
                               const void* v_pool, const int* block_table, int max_blocks,
                               const int* positions, const int* req_of_token, int n_tokens,
                               int n_heads, int n_kv, int hd, int block_size, float scale,
                               int window, float softcap, long long n_pages, const float* sink,
                               const float* slopes, int keep_first, long long out_stride,
                               int chunk, const int* cu_q, int longest, int shortest,
                               cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (hd > MOST_HD || hd <= 0 || n_heads % n_kv) return MLS_ERR_UNSUPPORTED;
    if (out_stride <= 0) out_stride = (long long)n_heads * hd;
    // requests of several tokens by tiles: heads of whole quads, up to 128 entries, at addresses that
    // can be read four entries at a time (a page's row then can, too)
    const uintptr_t bytes = dtype == MLS_BF16 ? 8 : 16;
    const bool tiles = cu_q && longest >= TILE_LEN && hd % 4 == 0 && hd <= 128 &&
                       (reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(k_pool) |
                        reinterpret_cast<uintptr_t>(v_pool)) % bytes == 0 && n_kv <= 1024 && n_heads <= 32768;
    if (tiles) {
#define TILE_GO(T, HD)                                                                             \
    launch_tile<T, HD>(qkv, out, k_pool, v_pool, block_table, max_blocks, positions, req_of_token, \
                       n_tokens, n_heads, n_kv, hd, block_size, scale, window, softcap, n_pages,   \
                       sink, slopes, keep_first, out_stride, window > 0 ? 0 : chunk, cu_q, stream)
        const int rc = dtype == MLS_BF16 ? (hd <= 64 ? TILE_GO(__nv_bfloat16, 64) : TILE_GO(__nv_bfloat16, 128))
                                         : (hd <= 64 ? TILE_GO(float, 64) : TILE_GO(float, 128));
#undef TILE_GO
        if (rc || shortest >= TILE_LEN) return rc;
    }
    const long long units = (long long)n_tokens * n_heads;
    const int blocks = (int)((units + WARPS - 1) / WARPS);
#define SIMT_GO(T, HD, SHORT)                                                                     \
    MLS_LAUNCH((attention_simt_kernel<T, HD, SHORT>), dim3(blocks), dim3(WARPS * 32), 0, stream,   \
               (const T*)qkv, (T*)out, (const T*)k_pool, (const T*)v_pool, block_table, max_blocks, \
               positions, req_of_token, n_tokens, n_heads, n_kv, hd, block_size, scale, window,    \
               softcap, n_pages, sink, slopes, keep_first, out_stride, window > 0 ? 0 : chunk, cu_q)
    if (tiles) {                                         // (heads of up to 128)
        if (dtype == MLS_BF16) SIMT_GO(__nv_bfloat16, 512, true);
        else SIMT_GO(float, 512, true);
    } else if (dtype == MLS_BF16) {
        if (hd <= 512) SIMT_GO(__nv_bfloat16, 512, false);
        else SIMT_GO(__nv_bfloat16, MOST_HD, false);
    } else {
        if (hd <= 512) SIMT_GO(float, 512, false);
        else SIMT_GO(float, MOST_HD, false);
    }
#undef SIMT_GO
    return launch_status();
}
