// The gated delta rule chunk by chunk for prompts of bfloat16 models (delta_rule.cu: token by token).
//
// Token by token a request's scan is a chain of 0.29 us a token.  Within a chunk of 64 tokens that starts from
// state S0, with G_t the product of the decays up to t, the values written are
//
//     u_t = b_t (v_t - G_t S0^T k_t) - sum_{s < t} L_ts u_s,        L_ts = b_t (G_t / G_s) k_t . k_s
//
// that is U = R + T R with R_t = b_t (v_t - G_t S0^T k_t) and 1 + T the inverse of 1 + L, which does not depend on
// the state (without the unit diagonal, so that the product's roundings count for the smaller share of U); and with P_ts = (G_t / G_s) q_t . k_s for s <= t
//
//     o_t = G_t S0^T q_t + sum_s P_ts u_s                 S0' = G_C S0 + sum_s (G_C / G_s) k_s u_s^T
//
//   delta_chunk_prep   for every chunk and key head at once: q and k as bfloat16 parts (bf16_parts.cuh) in the layout
//                      that shared memory takes them in, q k^T and k k^T in one product of 128 rows, and for every
//                      value head that shares the key head P, T (16 x 16 blocks inverted by forward substitution,
//                      the blocks below by products) and the factors b_t, G_t, G_C / G_t
//   delta_chunk_scan   a block a request, value head and 128 columns of the state walks the chunks: five products
//                      a chunk on the tensor cores, the columns on the 128-row side, from tensor memory
//
// A thread of the scan owns half of a column of the state (its lane of tensor memory, half of the rows) in registers
// and half of the tokens of R, U and o; S0, R and U go into tensor memory as parts, K, Q, T and P come from
// shared memory (K serves as K-major operand for S0^T k and as MN-major one for sum k u^T), copied ahead by
// a warp of its own.  Ratios G_t / G_s come from differences of float64 sums of logarithms, never from a
// quotient.  Accumulators hold at most 64 of k (P U: 32, q k^T and k k^T: 16), small products first.
//
// A value that is infinite or not a number counts as zero for the tokens before it; from its token on the
// column's outputs and state are no numbers (token by token they are not finite from there on either).
//
// What bounds the scan: a chunk's chain, 10,600 cycles (rows of 128): S0 into tensor memory 1,000, its products
// 1,500 (under them the outputs before leave and the values come), R 1,400, T R 800, U twice 1,700, the state's
// product 900 more and its sum 250, P U 800, and the hand-overs.  What bounds the preparation: loads of rows all blocks
// ask for at once 8,000 cycles of 40,000, the ratios 4,000 and T 5,500 a value head.
//
// Measured (the two kernels together against token by token): 32 heads of 128 x 128, requests of 341 and 683 tokens
// 202 -> 108 us, one of 2,048 389 -> 276.  Products issued by a warp that also owns
// columns held it up for 3,700 cycles a chunk (181 us for the first).  Distance from float64 as a multiple of token by
// token's (2-norms over all outputs; 8 to 32 heads of 64 x 128 to 128 x 256, 256 to 1,501 tokens, six seeds): outputs 0.91 to
// 1.09, 0.99 on average (heads of 64 0.94, of 96 0.97, of 128 1.02), states 0.59 to 0.72.  With q k^T and k k^T over 32 and
// expf's ratios outputs 0.94 to 1.11 (1.01), states 0.61 to 0.75, 3 us less; with q S0 in four accumulators of 32 instead
// of two of 64 outputs 0.91 to 1.07 (0.98), 12 us more; T R over 32 and P U over 16 change nothing.
#include "bf16_parts.cuh"
#include "chunk_common.cuh"
#include "delta_rule.h"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace mls_delta {
namespace {
using mls_chunk::Args;
using mls_chunk::C;
using mls_chunk::locate;
using mls_chunk::Part;
using mls_chunk::Where;
using namespace mls_tc;
using namespace mls_tma;

constexpr int TILE = C * 128;                          // bytes of 64 rows of 64 bfloat16
constexpr int UMMA_K = 16;
constexpr int FACTORS = 4 * C;                         // floats of a chunk and value head: b, G_t, G_C / G_t, (G_C)

// Scratch of a part: every chunk's and key head's k and q tiles, its value heads' P, T and factors.
struct Place {
    uint8_t* base;
    int H, G, e_tiles;
    __host__ __device__ size_t head_bytes() const { return 2 * 3 * TILE + FACTORS * 4; }
    __host__ __device__ size_t key_bytes() const { return (size_t)e_tiles * 2 * 3 * TILE; }
    __host__ __device__ size_t chunk_bytes() const { return H * head_bytes() + G * key_bytes(); }
    // [tile of 64 of e][part] of k, then of q
    __device__ uint8_t* k(size_t chunk, int kv) const { return base + chunk * chunk_bytes() + kv * key_bytes(); }
    __device__ uint8_t* q(size_t chunk, int kv) const { return k(chunk, kv) + (size_t)e_tiles * 3 * TILE; }
    // [part] of P, of T, then the factors
    __device__ uint8_t* P(size_t chunk, int head) const {
        return base + chunk * chunk_bytes() + G * key_bytes() + head * head_bytes();
    }
    __device__ uint8_t* T(size_t chunk, int head) const { return P(chunk, head) + 3 * TILE; }
    __device__ float* factors(size_t chunk, int head) const {
        return reinterpret_cast<float*>(P(chunk, head) + 2 * 3 * TILE);
    }
};

// Where entries x .. x + 3 of row r lie in a tile (the 128-byte swizzle).
__device__ __forceinline__ int swizzled(int r, int x) { return r * 128 + (((x >> 3) ^ (r & 7)) << 4) + (x & 7) * 2; }
__device__ __forceinline__ uint2 part4(float4& v) {
    uint2 two;
    two.x = bf16_part_up(v.x, v.y);
    two.y = bf16_part_up(v.z, v.w);
    return two;
}
// exp(d) for a float64 d <= 0, rounded once (expf's own 2 ulp showed in outputs and states).
__device__ __forceinline__ float exp_of(double d) { return (float)exp(d); }

constexpr int PREP_THREADS = 256, PAD = C + 4, MAX_RATIO = 4;

__global__ void __launch_bounds__(PREP_THREADS, 2)
delta_chunk_prep_kernel(const ChunkArgs a, const __grid_constant__ Args where, const Part part, const Place to) {
    chain_wait();
    Where w;
    if (!locate<false>(where, part, blockIdx.x, w)) return;
    extern __shared__ uint8_t smem_raw[];
    __shared__ double F_s[MAX_RATIO][C];
    __shared__ float beta_s[MAX_RATIO][C];
    __shared__ __align__(8) uint64_t bar_s;
    __shared__ uint32_t tmem_slot_s;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u, bar = smem_u32(&bar_s);
    uint8_t* tiles = smem_raw + (base - raw);          // [tile of e][part][q | k]: 128 rows of one operand
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31, tid = threadIdx.x;
    const int kv = blockIdx.y, ratio = a.H / a.G;
    if (tid == 0) {
        mbar_init(bar, 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_slot_s), 256);
        chain_release();                 // (not before: see there)
    }
    const Prepared rows(a.n_tokens, a.H, a.G, a.er, a.fr);
    // q and k as parts, to shared memory for their products and to scratch for the scan
    {
        const float* src = a.rows + rows.qk(kv, w.t0);
        uint8_t *k_to = to.k(w.idx, kv), *q_to = to.q(w.idx, kv);
        constexpr int AHEAD = 4;
        const int quads = to.e_tiles * C * 16;         // of q, and as many of k
        for (int u0 = tid; u0 < 2 * quads; u0 += AHEAD * PREP_THREADS) {
            float4 v[AHEAD];
#pragma unroll
            for (int y = 0; y < AHEAD; ++y) {
                const int u = u0 + y * PREP_THREADS, is_k = u >= quads, r = u - is_k * quads;
                const int tile = r / (C * 16), t = (r / 16) % C, x = 64 * tile + 4 * (r % 16);
                v[y] = u < 2 * quads && t < w.n && x < a.er
                           ? *reinterpret_cast<const float4*>(src + (size_t)t * 2 * a.er + is_k * a.er + x)
                           : make_float4(0.f, 0.f, 0.f, 0.f);
            }
#pragma unroll
            for (int y = 0; y < AHEAD; ++y) {
                const int u = u0 + y * PREP_THREADS, is_k = u >= quads, r = u - is_k * quads;
                if (u >= 2 * quads) break;
                const int tile = r / (C * 16), at = swizzled((r / 16) % C, 4 * (r % 16));
                uint8_t* dst = (is_k ? k_to : q_to) + (size_t)tile * 3 * TILE + at;
                uint8_t* own = tiles + tile * 6 * TILE + is_k * TILE + at;
#pragma unroll
                for (int p = 0; p < 3; ++p) {
                    const uint2 two = part4(v[y]);
                    *reinterpret_cast<uint2*>(dst + p * TILE) = two;
                    *reinterpret_cast<uint2*>(own + p * 2 * TILE) = two;
                }
            }
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
    bool timed_out = false;
    // sums of the decays' logarithms of value heads h0 .. h0 + 3, a warp of the last four each, two tokens a lane
    // (past the chunk's end nothing decays)
    auto decays = [&](int h0) {
        const int own = warp - 4;
        if (own < 0 || h0 + own >= ratio) return;
        const int head = kv * ratio + h0 + own;
        double l[2];
#pragma unroll
        for (int x = 0; x < 2; ++x) {
            const int t = 2 * lane + x;
            const float* s = a.rows + rows.scalars(head, w.t0 + min(t, w.n - 1));
            const float g = s[0];
            l[x] = t < w.n ? (g >= 1e-38f ? log((double)g) : g >= 0.f ? -1e4 : (double)g * NAN) : 0.0;
            beta_s[own][t] = t < w.n ? s[1] : 0.f;
        }
        l[1] += l[0];
        double sum = l[1];
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const double x = __shfl_up_sync(0xffffffffu, sum, o);
            if (lane >= o) sum += x;
        }
        F_s[own][2 * lane] = l[0] + (sum - l[1]);
        F_s[own][2 * lane + 1] = sum;
    };
    // q k^T and k k^T, 16 of e an accumulator, a tile of e at a time
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    float sum[C];
#pragma unroll
    for (int x = 0; x < C; ++x) sum[x] = 0.f;
    for (int tile = 0; tile < to.e_tiles; ++tile) {
        if (tile) {                                    // the sums of the tile before have been read
            tc_fence_before();
            __syncthreads();
            tc_fence_after();
        }
        if (warp == 0) {
            if (elect_one()) {
                constexpr uint32_t idesc = umma_idesc(C);
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    const uint32_t d = tmem + kk * C, at = base + tile * 6 * TILE + kk * UMMA_K * 2;
                    // part x of [q; k] times part y of k; the first of the next kind divides what is there
                    auto qk = [&](int x) { return umma_desc(at + x * 2 * TILE); };
                    auto k = [&](int y) { return umma_desc(at + (y * 2 + 1) * TILE); };
                    umma(d, qk(1), k(1), idesc, 0);
                    umma(d, qk(0), k(2), idesc, 1);
                    umma(d, qk(2), k(0), idesc, 1);
                    umma_onto<PART_SHIFT>(d, qk(0), k(1), idesc);
                    umma(d, qk(1), k(0), idesc, 1);
                    umma_onto<PART_SHIFT>(d, qk(0), k(0), idesc);
                }
                umma_commit(bar);
            }
            __syncwarp();
        }
        if (tile == 0) decays(0);
        if (!timed_out && !mbar_wait(bar, tile & 1)) timed_out = true;
        tc_fence_after();
        if (warp < 4) {
#pragma unroll
            for (int c0 = 0; c0 < C; c0 += 16)
#pragma unroll
                for (int kk = 0; kk < 4; ++kk) {
                    uint32_t x[16];
                    tmem_ld16(tmem + lanes + kk * C + c0, x);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i) sum[c0 + i] += __uint_as_float(x[i]);
                }
        }
    }
    float* dots = reinterpret_cast<float*>(tiles);     // (all products are done: the tiles' room) [q k^T; k k^T]: [128][PAD]
    float* L = dots + 2 * C * PAD;                     // [64][PAD]
    float* T = L + C * PAD;                            // [64][PAD]
    float* M = T + C * PAD;                            // [3][16][20]
    if (warp < 4) {
        float* dst = dots + (warp * 32 + lane) * PAD;
#pragma unroll
        for (int i = 0; i < C; i += 4)
            *reinterpret_cast<float4*>(dst + i) = make_float4(sum[i], sum[i + 1], sum[i + 2], sum[i + 3]);
    }
    tc_fence_before();
    for (int h = 0; h < ratio; ++h) {
        const int head = kv * ratio + h;
        float* factors = to.factors(w.idx, head);
        const double* F = F_s[h % MAX_RATIO];
        const float* beta = beta_s[h % MAX_RATIO];
        if (h && h % MAX_RATIO == 0) {
            __syncthreads();
            decays(h);
        }
        __syncthreads();
        if (tid < C) {
            factors[tid] = beta[tid];
            factors[C + tid] = exp_of(F[tid]);
            factors[2 * C + tid] = exp_of(F[C - 1] - F[tid]);
        }
        // P, and L
        uint8_t* P_to = to.P(w.idx, head);
#pragma unroll 1
        for (int u = tid; u < C * 16; u += PREP_THREADS) {
            const int t = u / 16, s0 = 4 * (u % 16);
            const double Ft = F[t];
            const float b = beta[t];
            float4 p = make_float4(0.f, 0.f, 0.f, 0.f), l = p;
            if (s0 <= t) {
                const float4 qk = *reinterpret_cast<const float4*>(dots + t * PAD + s0);
                const float4 kk = *reinterpret_cast<const float4*>(dots + (C + t) * PAD + s0);
                const float f0 = exp_of(Ft - F[s0]), f1 = s0 + 1 <= t ? exp_of(Ft - F[s0 + 1]) : 0.f,
                            f2 = s0 + 2 <= t ? exp_of(Ft - F[s0 + 2]) : 0.f, f3 = s0 + 3 <= t ? exp_of(Ft - F[s0 + 3]) : 0.f;
                // (what lies above the diagonal is zero whatever the products there are)
                p = make_float4(f0 * qk.x, s0 + 1 <= t ? f1 * qk.y : 0.f, s0 + 2 <= t ? f2 * qk.z : 0.f,
                                s0 + 3 <= t ? f3 * qk.w : 0.f);
                l = make_float4(s0 < t ? b * f0 * kk.x : 0.f, s0 + 1 < t ? b * f1 * kk.y : 0.f,
                                s0 + 2 < t ? b * f2 * kk.z : 0.f, s0 + 3 < t ? b * f3 * kk.w : 0.f);
            }
            *reinterpret_cast<float4*>(L + t * PAD + s0) = l;
            *reinterpret_cast<float4*>(T + t * PAD + s0) = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int y = 0; y < 3; ++y) *reinterpret_cast<uint2*>(P_to + y * TILE + swizzled(t, s0)) = part4(p);
        }
        __syncthreads();
        // T = (1 + L)^-1: the blocks on the diagonal, a column a thread
        if (tid < C) {
            const int b0 = tid & ~15, c = tid & 15;
            float x[16];
#pragma unroll
            for (int r = 0; r < 16; ++r) {
                float s = r == c ? 1.f : 0.f;
#pragma unroll
                for (int k = 0; k < r; ++k) s = fmaf(-L[(b0 + r) * PAD + b0 + k], x[k], s);
                x[r] = r < c ? 0.f : s;
                T[(b0 + r) * PAD + b0 + c] = x[r];
            }
        }
        // those below, diagonal after diagonal: T_ij = -T_ii sum_k L_ik T_kj; four columns a thread, a block of 16 x 16
        // 64 threads (an output a thread is bound by its reads of shared memory)
        const int block = tid >> 6, r = (tid >> 2) & 15, c4 = 4 * (tid & 3);
        // `lower`: the row's entries from n on are zeros that must not meet what is no number
        auto times_rows = [&](const float* row, const float* B, int apart, int n, bool lower, float4& sum) {
#pragma unroll 4
            for (int k = 0; k < n; k += 4) {              // (n rounded up to four)
                const float4 x = *reinterpret_cast<const float4*>(row + k);
                const float xs[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                for (int y = 0; y < 4; ++y) {
                    const float4 z = *reinterpret_cast<const float4*>(B + (k + y) * apart);
                    if (lower && k + y >= n) continue;
                    sum = make_float4(fmaf(xs[y], z.x, sum.x), fmaf(xs[y], z.y, sum.y), fmaf(xs[y], z.z, sum.z),
                                      fmaf(xs[y], z.w, sum.w));
                }
            }
        };
#pragma unroll 1
        for (int d = 1; d < 4; ++d) {
            const int j = block, i = j + d;
            __syncthreads();
            if (i < 4) {
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                times_rows(L + (16 * i + r) * PAD + 16 * j, T + 16 * j * PAD + 16 * j + c4, PAD, 16 * d, false, sum);
                *reinterpret_cast<float4*>(M + (j * 16 + r) * 20 + c4) = sum;
            }
            __syncthreads();
            if (i < 4) {
                float4 sum = make_float4(0.f, 0.f, 0.f, 0.f);
                times_rows(T + (16 * i + r) * PAD + 16 * i, M + j * 16 * 20 + c4, 20, r + 1, true, sum);
                *reinterpret_cast<float4*>(T + (16 * i + r) * PAD + 16 * j + c4) =
                    make_float4(-sum.x, -sum.y, -sum.z, -sum.w);
            }
        }
        __syncthreads();
        uint8_t* T_to = to.T(w.idx, head);
        for (int u = tid; u < C * 16; u += PREP_THREADS) {
            const int t = u / 16, s0 = 4 * (u % 16);
            float4 v = *reinterpret_cast<const float4*>(T + t * PAD + s0);
            v = make_float4(s0 == t ? 0.f : v.x, s0 + 1 == t ? 0.f : v.y, s0 + 2 == t ? 0.f : v.z, s0 + 3 == t ? 0.f : v.w);
#pragma unroll
            for (int y = 0; y < 3; ++y) *reinterpret_cast<uint2*>(T_to + y * TILE + swizzled(t, s0)) = part4(v);
        }
    }
    if (timed_out && a.status) atomicOr(a.status, MLS_STATUS_TIMEOUT);
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 256);
}

// ---------------------------------------------------------------------------------- scan
constexpr int SCAN_THREADS = 384;                      // eight warps of columns, one that copies ahead, one that multiplies

// ER: rows of the state (of 32 each).  Tensor memory: S0 as parts [0, 3 ER / 2), later U [0, 96); R, later the
// decayed U, later half of P U 96; S0^T q, half of the rows after the other, and half of P U 64; S0^T k (two of
// 64), T R and the state's sum 128.
template <int ER>
__global__ void __launch_bounds__(SCAN_THREADS, 1)
delta_chunk_scan_kernel(const ChunkArgs a, const __grid_constant__ Args where, const Part part, const Place from) {
    constexpr int E_TILES = (ER + 63) / 64, EH = ER / 2;
    constexpr int S_COL = 0, R_COL = 3 * ER / 2 < 96 ? 96 : 3 * ER / 2, O_COL = R_COL + 96, ACC = O_COL + 64;
    static_assert(ACC + 128 <= 512 && EH % 16 == 0 && EH <= 64, "tensor memory");
    constexpr int K_BYTES = E_TILES * 3 * TILE, Q_AT = 2 * K_BYTES, T_AT = Q_AT + K_BYTES, P_AT = T_AT + 3 * TILE,
                  F_AT = P_AT + 3 * TILE;
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<true>(where, part, blockIdx.z, w)) return;
    if (w.chunks <= 0) return;
    extern __shared__ uint8_t smem_raw[];
    __shared__ __align__(8) uint64_t bars[16];
    __shared__ uint32_t tmem_slot_s;
    __shared__ int dead_s[2][UMMA_M];                  // a column's first token that is no number
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    const float* factors_s = reinterpret_cast<const float*>(smem_raw + (base - raw) + F_AT);
    // copies landed; products done; operands in tensor memory: S0, R, the decayed U, U
    enum { K_FULL = 0, Q_FULL = 2, T_FULL, P_FULL, KS, QS, TR, QS2, KU, PU, S_PUT, R_PUT, O_READ, Z_PUT, U_PUT };
    auto bar = [&](int i) { return smem_u32(&bars[i]); };
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < 16; ++i) mbar_init(bar(i), 1);
        fence_barrier_init();
    }
    if (threadIdx.x < 2 * UMMA_M) dead_s[threadIdx.x / UMMA_M][threadIdx.x % UMMA_M] = C;
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_slot_s), 512);
        chain_release();                 // (not before: see there)
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
    const int kv = head / (a.H / a.G);
    bool timed_out = false;

    if (warp >= 8 && ER > 64) fewer_registers<72>();
    if (warp == 8) {
        // ------------------------------------------------------------------ copies ahead
        if (lane == 0) {
            auto load = [&](int full, uint32_t at, const void* src, uint32_t bytes) {
                bulk_load_1d(base + at, src, bytes, bar(full));
            };
            auto load_k = [&](int c) {
                const int b = c & 1;
                mbar_arrive_expect_tx(bar(K_FULL + b), K_BYTES + FACTORS * 4);
                load(K_FULL + b, b * K_BYTES, from.k(w.idx + c, kv), K_BYTES);
                load(K_FULL + b, F_AT + b * FACTORS * 4, from.factors(w.idx + c, head), FACTORS * 4);
            };
            auto load_q = [&](int c) {
                mbar_arrive_expect_tx(bar(Q_FULL), K_BYTES);
                load(Q_FULL, Q_AT, from.q(w.idx + c, kv), K_BYTES);
            };
            auto load_t = [&](int c) {
                mbar_arrive_expect_tx(bar(T_FULL), 3 * TILE);
                load(T_FULL, T_AT, from.T(w.idx + c, head), 3 * TILE);
            };
            auto load_p = [&](int c) {
                mbar_arrive_expect_tx(bar(P_FULL), 3 * TILE);
                load(P_FULL, P_AT, from.P(w.idx + c, head), 3 * TILE);
            };
            load_k(0);
            load_q(0);
            load_t(0);
            load_p(0);
            if (w.chunks > 1) load_k(1);
            int k_last = w.chunks > 1 ? 1 : 0, last = 0;
            for (int c = 0; c + 1 < w.chunks; ++c) {
                if (!mbar_wait(bar(TR), c & 1)) timed_out = true;
                load_t(c + 1);
                if (!mbar_wait(bar(QS2), c & 1)) timed_out = true;
                load_q(c + 1);
                // (PU ends behind U_PUT, ahead of which lies every read of the factors that come with k; behind KU alone
                // the columns may still read them, and KU may end once more before this warp looks: all that chunk
                // c + 1 needs for it is there)
                if (!mbar_wait(bar(PU), c & 1)) timed_out = true;
                load_p(c + 1);
                if (c + 2 < w.chunks) load_k(c + 2), k_last = c + 2;
                last = c + 1;
                if (timed_out) break;
            }
            // the copies under way land before the block's shared memory goes away
            for (int c = k_last > 0 ? k_last - 1 : 0; c <= k_last; ++c)
                if (!mbar_wait(bar(K_FULL + (c & 1)), (c >> 1) & 1)) timed_out = true;
            if (!mbar_wait(bar(Q_FULL), last & 1) || !mbar_wait(bar(T_FULL), last & 1) ||
                !mbar_wait(bar(P_FULL), last & 1))
                timed_out = true;
        }
    } else if (warp == 9) {
        // --------------------------------------------------------------------- products
        // (a warp of its own: the instructions are taken no faster than they run, 39 cycles each for 64 columns)
        auto wait = [&](int i, int parity) {
            if (!timed_out && !mbar_wait(bar(i), parity)) timed_out = true;
            tc_fence_after();
        };
        // D (+)= A as parts `apart` columns from each other times B's tiles of parts, K of [k0, k1) in steps of
        // 16, the small products first
        auto multiply = [&](uint32_t d, uint32_t A, int apart, uint32_t B, uint32_t idesc, int k0, int k1, bool mn) {
            uint32_t accumulate = 0;
            auto product = [&](int x, int y, bool next_kind) {      // (its first divides what is there)
                for (int kk = k0; kk < k1; ++kk) {
                    const uint64_t desc = mn ? umma_desc_mn(B + y * TILE + kk * UMMA_K * 128, 3 * TILE)
                                             : umma_desc(B + ((kk >> 2) * 3 + y) * TILE + (kk & 3) * 32);
                    if (next_kind && kk == k0) umma_ts_onto<PART_SHIFT>(d, A + x * apart + kk * 8, desc, idesc);
                    else umma_ts(d, A + x * apart + kk * 8, desc, idesc, accumulate);
                    accumulate = 1;
                }
            };
            product(1, 1, false);
            product(0, 2, false);
            product(2, 0, false);
            product(0, 1, true);
            product(1, 0, false);
            product(0, 0, true);
        };
        constexpr uint32_t id = umma_idesc(C), id_mn = umma_idesc(ER, 1);
        for (int c = 0; c < w.chunks; ++c) {
            const int ph = c & 1;
            const uint32_t k_tiles = base + ph * K_BYTES;
            wait(K_FULL + ph, (c >> 1) & 1);
            wait(S_PUT, ph);
            if (elect_one()) {
                multiply(tmem + ACC, tmem + S_COL, ER / 2, k_tiles, id, 0, EH / 16, false);
                multiply(tmem + ACC + C, tmem + S_COL, ER / 2, k_tiles, id, EH / 16, ER / 16, false);
                umma_commit(bar(KS));
            }
            __syncwarp();
            wait(Q_FULL, ph);
            if (elect_one()) {
                multiply(tmem + O_COL, tmem + S_COL, ER / 2, base + Q_AT, id, 0, EH / 16, false);
                umma_commit(bar(QS));
            }
            __syncwarp();
            wait(T_FULL, ph);
            wait(R_PUT, ph);
            if (elect_one()) {
                multiply(tmem + ACC, tmem + R_COL, 32, base + T_AT, id, 0, 4, false);
                umma_commit(bar(TR));
            }
            __syncwarp();
            // (behind T R, and under the threads' work on U)
            wait(O_READ, ph);
            if (elect_one()) {
                multiply(tmem + O_COL, tmem + S_COL, ER / 2, base + Q_AT, id, EH / 16, ER / 16, false);
                umma_commit(bar(QS2));
            }
            __syncwarp();
            wait(Z_PUT, ph);
            if (elect_one()) {
                multiply(tmem + ACC, tmem + R_COL, 32, k_tiles, id_mn, 0, 4, true);
                umma_commit(bar(KU));
            }
            __syncwarp();
            wait(P_FULL, ph);
            wait(U_PUT, ph);
            if (elect_one()) {
                multiply(tmem + O_COL, tmem + S_COL, 32, base + P_AT, id, 0, 2, false);
                multiply(tmem + R_COL, tmem + S_COL, 32, base + P_AT, id, 2, 4, false);
                umma_commit(bar(PU));
            }
            __syncwarp();
        }
    } else if (warp < 8) {
        // ----------------------------------------------------------------------- columns
        if (ER > 64) more_registers<216>();
        const int half = warp >> 2, row = (warp & 3) * 32 + lane;
        const int column = blockIdx.x * UMMA_M + row, j = min(column, a.fr - 1);
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        const Prepared rows(a.n_tokens, a.H, a.G, ER, a.fr);
        // all columns' operands are in tensor memory
        auto hand_over = [&](int i) {
            tmem_st_wait();
            tc_fence_before();
            asm volatile("bar.sync 1, 256;\n" ::: "memory");
            if (threadIdx.x == 0) mbar_arrive(bar(i));
        };
        auto wait = [&](int i, int parity) {
            if (!timed_out && !mbar_wait(bar(i), parity)) timed_out = true;
            tc_fence_after();
        };
        float* S_at = a.state + (size_t)a.state_slot[w.r] * a.state_stride + ((size_t)head * a.fr + j) * ER + half * EH;
        float S[EH];
#pragma unroll
        for (int i = 0; i < EH; i += 4) {
            const float4 v = *reinterpret_cast<const float4*>(S_at + i);
            S[i] = v.x, S[i + 1] = v.y, S[i + 2] = v.z, S[i + 3] = v.w;
        }
        const int t_end = a.cu_q[w.r + 1];
        if (part.first == 0) {
            // the convolution's last inputs (the preparation has read the older ones)
            const int t_begin = a.cu_q[w.r], blocks = gridDim.x * gridDim.y;
            float* ring = a.state + (size_t)a.state_slot[w.r] * a.state_stride + a.ring_at;
            for (int t = max(t_begin, t_end - (a.taps - 1)); t < t_end; ++t) {
                float* dst = ring + (size_t)(a.positions[t] % a.taps) * a.channels;
                for (int i = (blockIdx.y * gridDim.x + blockIdx.x) * 256 + threadIdx.x; i < a.channels; i += blocks * 256)
                    dst[i] = a.proj[(size_t)t * a.width + a.qkv_col + i];
            }
        }
        float v[32];
        auto load_v = [&](int c) {                      // this thread's 32 tokens of chunk c
            const int t0 = w.t0 + c * C + 32 * half;
            const float* src = a.rows + rows.v(head, j / DR_COLS, t0) + j % DR_COLS;
#pragma unroll
            for (int x = 0; x < 32; ++x) v[x] = t0 + x < t_end ? src[x * DR_COLS] : 0.f;
        };
        // 16 entries as parts: into columns `at` of the parts, `apart` columns from part to part
        auto put16 = [&](uint32_t at, int apart, float (&x)[16]) {
#pragma unroll
            for (int y = 0; y < 3; ++y) {
                uint32_t two[8];
#pragma unroll
                for (int i = 0; i < 8; ++i) two[i] = bf16_part_up(x[2 * i], x[2 * i + 1]);
                tmem_st8(at + lanes + y * apart, two);
            }
        };
        // outputs of the chunk before, kept until the next products are under way
        float o[32];
        auto store = [&](int c) {
            const int t0 = w.t0 + c * C + 32 * half;
            const int n = column < a.f ? t_end - t0 : 0;
            float* dst = a.out + ((size_t)t0 * a.H + head) * a.f + column;
            const size_t apart = (size_t)a.H * a.f;
            if (n >= 32) {
#pragma unroll
                for (int x = 0; x < 32; ++x, dst += apart) *dst = o[x];
            } else {
#pragma unroll
                for (int x = 0; x < 32; ++x, dst += apart)
                    if (x < n) *dst = o[x];
            }
        };
        for (int c = 0; c < w.chunks; ++c) {
            const int ph = c & 1;
            const float* factors = factors_s + ph * FACTORS + 32 * half;
            // S0 as parts; S0^T k and S0^T q
#pragma unroll
            for (int i = 0; i < EH; i += 16) {
                float x[16];
#pragma unroll
                for (int y = 0; y < 16; ++y) x[y] = S[i + y];
                put16(tmem + S_COL + (half * EH + i) / 2, ER / 2, x);
            }
            hand_over(S_PUT);
            load_v(c);
            if (c > 0) store(c - 1);
            // R
            wait(K_FULL + ph, (c >> 1) & 1);             // (the factors came with k)
            wait(KS, ph);
            float u[32];
            int odd = C;
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                uint32_t p[16], q[16];
                tmem_ld16(tmem + ACC + lanes + 32 * half + x0, p);
                tmem_ld16(tmem + ACC + C + lanes + 32 * half + x0, q);
                tmem_ld_wait();
                float any = 0.f;
                float R[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    const float sk = __uint_as_float(p[x]) + __uint_as_float(q[x]);
                    R[x] = factors[x0 + x] * fmaf(-factors[C + x0 + x], sk, v[x0 + x]);
                    any = fmaf(R[x], 0.f, any);
                }
                if (any != 0.f) {
#pragma unroll
                    for (int x = 0; x < 16; ++x)
                        if (!finite(R[x])) {
                            odd = min(odd, 32 * half + x0 + x);
                            R[x] = 0.f;
                        }
                }
#pragma unroll
                for (int x = 0; x < 16; ++x) u[x0 + x] = R[x];
                put16(tmem + R_COL + (32 * half + x0) / 2, 32, R);
            }
            if (odd < C) atomicMin(&dead_s[ph][row], odd);
            hand_over(R_PUT);
            const int dead = dead_s[ph][row];
            dead_s[ph ^ 1][row] = C;                     // (both halves: for the next chunk)
            // what the state before the chunk gives to the outputs
            wait(QS, ph);
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                uint32_t p[16];
                tmem_ld16(tmem + O_COL + lanes + 32 * half + x0, p);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x) o[x0 + x] = __uint_as_float(p[x]);
            }
            hand_over(O_READ);
            // U: decayed to the chunk's end for the state, as it is for the outputs
            wait(TR, ph);
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                uint32_t p[16];
                tmem_ld16(tmem + ACC + lanes + 32 * half + x0, p);
                tmem_ld_wait();
                float z[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    u[x0 + x] = 32 * half + x0 + x < dead ? u[x0 + x] + __uint_as_float(p[x]) : 0.f;
                    z[x] = factors[2 * C + x0 + x] * u[x0 + x];
                }
                put16(tmem + R_COL + (32 * half + x0) / 2, 32, z);
            }
            const float whole = (factors_s + ph * FACTORS)[C + C - 1];
            hand_over(Z_PUT);
            wait(QS2, ph);
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                uint32_t p[16];
                tmem_ld16(tmem + O_COL + lanes + 32 * half + x0, p);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x)
                    o[x0 + x] = factors[C + x0 + x] * (o[x0 + x] + __uint_as_float(p[x]));
            }
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                float z[16];
#pragma unroll
                for (int x = 0; x < 16; ++x) z[x] = u[x0 + x];
                put16(tmem + S_COL + (32 * half + x0) / 2, 32, z);
            }
            hand_over(U_PUT);
            // the state behind the chunk
            wait(KU, ph);
#pragma unroll
            for (int i = 0; i < EH; i += 16) {
                uint32_t p[16];
                tmem_ld16(tmem + ACC + lanes + half * EH + i, p);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x) S[i + x] = fmaf(whole, S[i + x], __uint_as_float(p[x]));
            }
            if (dead < C)
#pragma unroll
                for (int i = 0; i < EH; ++i) S[i] = NAN;
            wait(PU, ph);
#pragma unroll
            for (int x0 = 0; x0 < 32; x0 += 16) {
                uint32_t p[16], q[16];
                tmem_ld16(tmem + O_COL + lanes + 32 * half + x0, p);
                tmem_ld16(tmem + R_COL + lanes + 32 * half + x0, q);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x)
                    o[x0 + x] = 32 * half + x0 + x < dead
                                    ? o[x0 + x] + (__uint_as_float(p[x]) + __uint_as_float(q[x])) : NAN;
            }
        }
        store(w.chunks - 1);
        if (column < a.fr)
#pragma unroll
            for (int i = 0; i < EH; i += 4)
                *reinterpret_cast<float4*>(S_at + i) = make_float4(S[i], S[i + 1], S[i + 2], S[i + 3]);
    }
    if (timed_out && a.status) atomicOr(a.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, 512);
}

template <int ER>
int launch_scan(const ChunkArgs& a, const Args& where, const Part& part, const Place& place, cudaStream_t stream) {
    constexpr int E_TILES = (ER + 63) / 64;
    const int smem = 3 * E_TILES * 3 * TILE + 2 * 3 * TILE + 2 * FACTORS * 4 + 1024;
    const int rc = (int)cudaFuncSetAttribute(delta_chunk_scan_kernel<ER>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
    if (rc) return rc;
    MLS_LAUNCH((delta_chunk_scan_kernel<ER>), dim3((a.fr + UMMA_M - 1) / UMMA_M, a.H, part.count), dim3(SCAN_THREADS),
               smem, stream, a, where, part, place);
    return launch_status();
}
}  // namespace

// Three blocks of 32 to four of the state's rows, and enough columns for the instruction's 128 rows.
bool chunk_fits(int er, int fr) { return er >= 64 && er <= 128 && fr >= 64; }

long long chunk_floats(int H, int G, int er) {
    const Place p{nullptr, H, G, (er + 63) / 64};
    return (long long)(p.chunk_bytes() / 4);
}

int chunk_scan(const ChunkArgs& a, float* scratch, cudaStream_t stream) {
    if (a.count <= 0 || a.span <= 0 || a.chunks <= 0) return 0;
    if (!chunk_fits(a.er, a.fr) || a.count > 65535 || a.H > 65535 || a.G > 65535 || a.least < 1 || a.from < 0 || a.first < 0 ||
        reinterpret_cast<uintptr_t>(scratch) % 16)
        return MLS_ERR_UNSUPPORTED;
    Args where{};
    where.cu_q = a.cu_q;
    where.n_requests = a.n_requests;
    where.least = a.least;
    const Part part{a.from, a.count, a.first, a.span, a.chunks};
    const Place place{reinterpret_cast<uint8_t*>(scratch), a.H, a.G, (a.er + 63) / 64};
    const int smem = place.e_tiles * 6 * TILE + 1024;
    const int need = 1024 + (4 * C * PAD + 3 * 16 * 20) * (int)sizeof(float);
    const int rc = (int)cudaFuncSetAttribute(delta_chunk_prep_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             smem > need ? smem : need);
    if (rc) return rc;
    MLS_LAUNCH((delta_chunk_prep_kernel), dim3(a.chunks, a.G), dim3(PREP_THREADS), smem > need ? smem : need, stream, a,
               where, part, place);
    const int launched = launch_status();
    if (launched) return launched;
    if (a.er == 64) return launch_scan<64>(a, where, part, place, stream);
    if (a.er == 96) return launch_scan<96>(a, where, part, place, stream);
    return launch_scan<128>(a, where, part, place, stream);
}
}  // namespace mls_delta
