// Routed experts: choose, sort, multiply expert by expert, add up.
//
// mls_route_topk: scores s = sigmoid(z), or softmax(z) over all outputs, of float32 router
//   logits z [T, E], or (mode 2) the logits plus a bias themselves, whose softmax over the chosen
//   ones gives the weights; for every token the `top` largest scores (plus a per-output correction
//   that enters the choice only; the lowest index wins a tie) with the scores themselves as
//   weights (optionally divided by their sum + renorm_eps).  With n_groups > 1 the outputs form
//   n_groups equal groups of neighbours; a group's score is the sum of its two largest choice
//   scores, and only outputs of the keep_groups best groups (lowest index on a tie) can be
//   chosen.  A (token, choice) pair is a "slot": slot = t * top + j.  Outputs n_real .. E-1 stand for experts without weights that
//   return their input: they get no tiles, and mls_expert_combine adds weight * h for them.
// mls_route_sort: slots ordered by expert: order[p] = slot, offsets[E + 1], and the list
//   of row tiles (tile_expert, tile_row0) the CUDA-core products below walk.  One CTA.
// mls_expert_glu: y[p, :] = unit(Wg[e] a, Wu[e] a) with unit(g, u) = silu(g) * u or, with a
//   limit > 0, g' * sigmoid(alpha g') * (u' + 1), g' = min(g, limit), u' = clamp(u, +-limit);
//   a = weight[slot] * h[token]
//   (input scaling: the weight multiplies what enters the expert) or a = h[token]
//   (output scaling, applied by the down product instead).
// mls_expert_relu2: y[p, :] = relu(Wu[e] a)^2, experts without a gate.
// mls_expert_down: per_slot[slot, :] = Wd[e] y[p, :] (times the weight with output
//   scaling), float32.
// mls_expert_combine: delta[t] = sum_j per_slot[t * top + j] + shared[t], j ascending (shared: a
//   tensor, or the float32 K-parts of its product, shared_stride apart, added in their order); with a
//   gate (float32, one number a token) the shared addend is multiplied by sigmoid(gate[t]).
//
// The products run with float32 accumulation over k ascending: bfloat16 rows of whole
// 16-byte pieces on the tensor cores (experts_tc.cu), everything else on CUDA cores, one row
// tile of one expert a CTA; every row is computed by itself, so a token's result does
// not depend on the batch, on its place in the sorted order or on the other tokens of
// its expert.
#include "common.cuh"
#include "experts.h"

namespace {
using namespace mls_experts;
constexpr int BM = 32, BN = 64, BK = 32, TM = 2, TN = 4;   // 256 threads

constexpr int MAX_GROUPS = 256;

// HELD: outputs a lane keeps in registers (0: any number of outputs, none kept).
template <int HELD>
__global__ void route_topk_kernel(const float* __restrict__ logits, int logit_stride, int n_tokens,
                                  int n_experts, int top, int renorm, int mode,
                                  const float* __restrict__ correction, float renorm_eps,
                                  int n_groups, int keep_groups,
                                  int* __restrict__ idx, float* __restrict__ weight) {
    chain_release();
    chain_wait();
    // one warp a token
    __shared__ float group_score[4][MAX_GROUPS];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int t = blockIdx.x * (blockDim.x >> 5) + warp;
    if (t >= n_tokens) return;
    const float* z = logits + (size_t)t * logit_stride;
    const bool softmax = mode == 1, by_logit = mode == 2;     // (else sigmoid)
    // softmax over all outputs: the largest logit and the sum of exponentials, both in the
    // order of the lanes' strides, so a token's scores do not depend on its batch
    float z_max = 0.f, inv_sum = 1.f;
    if (softmax) {
        z_max = -INFINITY;
        for (int e = lane; e < n_experts; e += 32) z_max = fmaxf(z_max, z[e]);
        z_max = warp_max(z_max);
        float sum = 0.f;
        for (int e = lane; e < n_experts; e += 32) sum += expf(z[e] - z_max);
        inv_sum = 1.0f / warp_sum(sum);
    }
    // (in mode 2 the correction is a bias of the logits: part of the score)
    auto score = [&](int e) {
        if (by_logit) return correction ? z[e] + correction[e] : z[e];
        return softmax ? expf(z[e] - z_max) * inv_sum : 1.0f / (1.0f + expf(-z[e]));
    };
    const int group_size = n_groups > 1 ? n_experts / n_groups : n_experts;
    if (n_groups > 1) {
        // a group's score: the sum of its two largest choice scores (one, if it has one member)
        for (int g = lane; g < n_groups; g += 32) {
            float a = -INFINITY, b = -INFINITY;
            for (int e = g * group_size; e < (g + 1) * group_size; ++e) {
                const float s = score(e);
                const float c = (correction && !by_logit) ? s + correction[e] : s;
                if (c > a) { b = a; a = c; } else if (c > b) { b = c; }
            }
            group_score[warp][g] = group_size > 1 ? a + b : a;
        }
        __syncwarp();
    }
    // whether an output's group is among the kept ones: how many groups come before it
    auto kept = [&](int e) {
        const int g = e / group_size;
        const float mine = group_score[warp][g];
        int before = 0;
        for (int o = 0; o < n_groups; ++o) {
            const float other = group_score[warp][o];
            before += (other > mine || (other == mine && o < g)) ? 1 : 0;
        }
        return before < keep_groups;
    };
    // a lane's outputs lane, lane + 32, ...: their scores stay in registers where there are few (every
    // choice used to work all scores out again and read back what was chosen before)
    float score_r[HELD > 0 ? HELD : 1];
    unsigned gone = 0;                        // bit x: output lane + 32 x cannot be chosen (any more)
    if (HELD > 0) {
#pragma unroll
        for (int x = 0; x < HELD; ++x) {
            const int e = lane + 32 * x;
            score_r[x] = e < n_experts ? score(e) : 0.f;
            if (e >= n_experts || (n_groups > 1 && !kept(e))) gone |= 1u << x;
        }
    }
    float total = 0.f;
    for (int j = 0; j < top; ++j) {
        float best = -INFINITY, best_s = 0.f;
        int arg = 0x7fffffff;
        auto offer = [&](int e, float s) {
            const float c = (correction && !by_logit) ? s + correction[e] : s;      // the choice's score
            if (c > best || (c == best && e < arg)) {
                best = c;
                best_s = s;
                arg = e;
            }
        };
        if (HELD > 0) {
#pragma unroll
            for (int x = 0; x < HELD; ++x)
                if (!((gone >> x) & 1u)) offer(lane + 32 * x, score_r[x]);
        } else {
            for (int e = lane; e < n_experts; e += 32) {
                bool taken = n_groups > 1 && !kept(e);
                for (int p = 0; p < j; ++p) taken |= idx[(size_t)t * top + p] == e;
                if (!taken) offer(e, score(e));
            }
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ob = __shfl_xor_sync(0xffffffffu, best, o);
            const float os = __shfl_xor_sync(0xffffffffu, best_s, o);
            const int oa = __shfl_xor_sync(0xffffffffu, arg, o);
            if (ob > best || (ob == best && oa < arg)) {
                best = ob;
                best_s = os;
                arg = oa;
            }
        }
        if (arg >= n_experts) {                  // only scores that are not numbers were left
            arg = 0;
            best_s = 0.f;
        }
        if (HELD > 0 && (arg & 31) == lane) gone |= 1u << (arg >> 5);
        if (lane == 0) {
            idx[(size_t)t * top + j] = arg;
            weight[(size_t)t * top + j] = best_s;
        }
        total += best_s;
        __syncwarp();
    }
    if (by_logit) {
        // the first chosen logit is the largest
        if (lane == 0) {
            float* w = weight + (size_t)t * top;
            const float most = w[0];
            float sum = 0.f;
            for (int j = 0; j < top; ++j) sum += expf(w[j] - most);
            for (int j = 0; j < top; ++j) w[j] = expf(w[j] - most) / sum;
        }
        return;
    }
    if (renorm && lane == 0)
        for (int j = 0; j < top; ++j) weight[(size_t)t * top + j] /= total + renorm_eps;
}

// One block.  The counters lie in shared memory where they fit (SORT_SHARED), else in `cursor`; one
// warp scans them.  (Counters in global memory and one thread that walked the experts: 30 -> 12 us
// for 12,288 slots of 64 experts.)
constexpr int SORT_SHARED = 8192;
__global__ void __launch_bounds__(1024)
route_sort_kernel(const int* __restrict__ idx, int n_slots, int n_experts, int n_real,
                  int* __restrict__ order, int* __restrict__ offsets,
                  int* __restrict__ tile_expert, int* __restrict__ tile_row0, int max_tiles,
                  int* cursor /* [E] scratch */) {
    chain_release();
    extern __shared__ int count_s[];
    __shared__ int tiles_s;
    int* count = n_experts <= SORT_SHARED ? count_s : cursor;
    chain_wait();
    for (int e = threadIdx.x; e < n_experts; e += blockDim.x) count[e] = 0;
    __syncthreads();
    for (int s = threadIdx.x; s < n_slots; s += blockDim.x) atomicAdd(&count[idx[s]], 1);
    __syncthreads();
    if (threadIdx.x < 32) {
        int at = 0, tile = 0;                             // slots and tiles of the experts before
        const int lane = threadIdx.x;
        for (int e0 = 0; e0 < n_experts; e0 += 32) {
            const int e = e0 + lane;
            const int c = e < n_experts ? count[e] : 0;
            // (an expert past n_real has no weights: its slots are settled where the sum is taken)
            const int n = e < n_real ? (c + BM - 1) / BM : 0;
            int cs = c, ns = n;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int x = __shfl_up_sync(0xffffffffu, cs, o), y = __shfl_up_sync(0xffffffffu, ns, o);
                if (lane >= o) {
                    cs += x;
                    ns += y;
                }
            }
            if (e < n_experts) {
                offsets[e] = at + cs - c;
                count[e] = at + cs - c;
                for (int i = 0; i < n; ++i) {
                    const int k = tile + ns - n + i;
                    if (k >= max_tiles) break;
                    tile_expert[k] = e;
                    tile_row0[k] = at + cs - c + i * BM;
                }
            }
            at += __shfl_sync(0xffffffffu, cs, 31);
            tile += __shfl_sync(0xffffffffu, ns, 31);
        }
        if (lane == 0) {
            offsets[n_experts] = at;
            tiles_s = tile;
        }
    }
    __syncthreads();
    for (int k = tiles_s + threadIdx.x; k < max_tiles; k += blockDim.x) tile_expert[k] = -1;
    // which place a slot gets inside its expert is left to the atomics: every row is
    // computed by itself, so the values do not depend on it
    for (int s = threadIdx.x; s < n_slots; s += blockDim.x)
        order[atomicAdd(&count[idx[s]], 1)] = s;
}

// 16 bytes of a row as floats: eight bfloat16 or four float32.
template <typename T> struct Vec;
template <> struct Vec<float> {
    static constexpr int N = 4;
    static __device__ __forceinline__ void load(const float* p, float* out) {
        const float4 v = *reinterpret_cast<const float4*>(p);
        out[0] = v.x; out[1] = v.y; out[2] = v.z; out[3] = v.w;
    }
};
template <> struct Vec<__nv_bfloat16> {
    static constexpr int N = 8;
    static __device__ __forceinline__ void load(const __nv_bfloat16* p, float* out) {
        const uint4 raw = *reinterpret_cast<const uint4*>(p);
        const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&raw);
#pragma unroll
        for (int e = 0; e < 4; ++e) {
            const float2 f = __bfloat1622float2(h[e]);
            out[2 * e] = f.x;
            out[2 * e + 1] = f.y;
        }
    }
};

// Fill tile[k][row] (k < BK, row < ROWS) from rows of K-contiguous values: row r comes from
// src(r) (nullptr: zeros), scaled by scale(r).  16-byte loads where K allows them.
template <typename T, int ROWS, int PAD, typename Src>
__device__ __forceinline__ void fill_tile(float (*tile)[ROWS + PAD], int k0, int K, bool vec_ok,
                                          Src src) {
    constexpr int V = Vec<T>::N;
    if (vec_ok) {
        for (int u = threadIdx.x; u < ROWS * (BK / V); u += 256) {
            const int r = u / (BK / V), kv = (u - r * (BK / V)) * V;
            float scale = 1.f;
            const T* p = src(r, scale);
            float v[V];
            if (p && k0 + kv < K) {
                Vec<T>::load(p + k0 + kv, v);
            } else {
#pragma unroll
                for (int e = 0; e < V; ++e) v[e] = 0.f;
            }
#pragma unroll
            for (int e = 0; e < V; ++e) tile[kv + e][r] = v[e] * scale;
        }
    } else {
        for (int u = threadIdx.x; u < ROWS * BK; u += 256) {
            const int r = u / BK, k = u - r * BK;
            float scale = 1.f;
            const T* p = src(r, scale);
            tile[k][r] = (p && k0 + k < K) ? Elem<T>::load(p + k0 + k) * scale : 0.f;
        }
    }
}

// GATED: A row = h[slot / top] (* weight[slot] if scale), W = [gate rows | up rows] of
// expert e ([2F, K]), out y[p, n] = silu(gate) * up in T.
// RELU2: the same A row, W = Wu[e] ([F, K]), y[p, n] = relu(up)^2.
// DOWN: A row = y[p], W = Wd[e] ([N, K]), out per_slot[slot, n] float32 (* weight[slot]
// if scale).  A thread owns rows ty*TM.. and the columns tx, tx + 16, tx + 32, tx + 48.
template <typename T, int UNIT>
__global__ void __launch_bounds__(256)
expert_gemm_kernel(const T* __restrict__ A, const T* __restrict__ W, void* __restrict__ out,
                   const int* __restrict__ order, const int* __restrict__ offsets,
                   const int* __restrict__ tile_expert, const int* __restrict__ tile_row0,
                   const float* __restrict__ weight, int top, int scale, int N, int K,
                   float alpha, float limit) {
    constexpr bool GLU = UNIT == GATED, UP = UNIT != DOWN;
    chain_release();
    chain_wait();
    const int e = tile_expert[blockIdx.y];
    if (e < 0) return;
    __shared__ float As[BK][BM + 1];
    __shared__ float Ws[BK][BN + 1];
    __shared__ float Us[GLU ? BK : 1][BN + 1];
    __shared__ int slot_s[BM];
    const int tid = threadIdx.x;
    const int p0 = tile_row0[blockIdx.y], p_end = offsets[e + 1];
    const int n0 = blockIdx.x * BN;
    const int tx = tid % 16, ty = tid / 16;                     // 16 x 16
    if (tid < BM) slot_s[tid] = p0 + tid < p_end ? order[p0 + tid] : -1;
    __syncthreads();
    const T* We = W + (size_t)e * (GLU ? 2 : 1) * N * K;
    const bool vec_ok = K % Vec<T>::N == 0 &&
                        (reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) % 16 == 0;
    float acc[TM][TN], acu[GLU ? TM : 1][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            acc[i][j] = 0.f;
            if (GLU) acu[i][j] = 0.f;
        }
    for (int k0 = 0; k0 < K; k0 += BK) {
        fill_tile<T, BM, 1>(As, k0, K, vec_ok, [&](int r, float& sc) -> const T* {
            const int slot = slot_s[r];
            if (slot < 0) return nullptr;
            if (UP) {
                if (scale) sc = weight[slot];
                return A + (size_t)(slot / top) * K;
            }
            return A + (size_t)(p0 + r) * K;
        });
        fill_tile<T, BN, 1>(Ws, k0, K, vec_ok, [&](int r, float&) -> const T* {
            return n0 + r < N ? We + (size_t)(n0 + r) * K : nullptr;
        });
        if (GLU)
            fill_tile<T, BN, 1>(Us, k0, K, vec_ok, [&](int r, float&) -> const T* {
                return n0 + r < N ? We + (size_t)(N + n0 + r) * K : nullptr;
            });
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            float a[TM], w[TN], u[TN];
#pragma unroll
            for (int i = 0; i < TM; ++i) a[i] = As[kk][ty * TM + i];
#pragma unroll
            for (int j = 0; j < TN; ++j) {
                w[j] = Ws[kk][tx + 16 * j];
                if (GLU) u[j] = Us[kk][tx + 16 * j];
            }
#pragma unroll
            for (int i = 0; i < TM; ++i)
#pragma unroll
                for (int j = 0; j < TN; ++j) {
                    acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
                    if (GLU) acu[i][j] = fmaf(a[i], u[j], acu[i][j]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int r = ty * TM + i;
        const int slot = slot_s[r];
        if (slot < 0) continue;
#pragma unroll
        for (int j = 0; j < TN; ++j) {
            const int n = n0 + tx + 16 * j;
            if (n >= N) continue;
            if (GLU) {
                Elem<T>::store((T*)out + (size_t)(p0 + r) * N + n,
                               gated_unit(acc[i][j], acu[i][j], alpha, limit));
            } else if (UP) {
                const float u = fmaxf(acc[i][j], 0.f);
                Elem<T>::store((T*)out + (size_t)(p0 + r) * N + n, u * u);
            } else {
                ((float*)out)[(size_t)slot * N + n] = scale ? acc[i][j] * weight[slot] : acc[i][j];
            }
        }
    }
}

template <typename T>
__global__ void expert_combine_kernel(const float* __restrict__ per_slot, int top,
                                      const void* __restrict__ shared, int shared_dtype,
                                      int shared_parts, size_t shared_stride,
                                      const int* __restrict__ idx, const float* __restrict__ weight,
                                      int n_real, const T* __restrict__ h,
                                      const float* __restrict__ gate, int gate_stride,
                                      T* __restrict__ delta, size_t n, int d) {
    chain_release();
    chain_wait();
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const size_t t = i / d, c = i - t * d;
        float s = 0.f;
        for (int j = 0; j < top; ++j) {
            // a choice past the experts that have weights returns its input, times its weight
            if (idx && idx[t * top + j] >= n_real)
                s += weight[t * top + j] * Elem<T>::load(h + i);
            else
                s += per_slot[(t * top + j) * d + c];
        }
        if (shared) {
            float v = load_as_float(shared, i, shared_dtype);
#pragma unroll 4
            for (int k = 1; k < shared_parts; ++k) v += ((const float*)shared)[i + k * shared_stride];
            s += gate ? times_sigmoid(v, gate[t * gate_stride]) : v;
        }
        Elem<T>::store(delta + i, s);
    }
}
// The same, four entries a thread, for rows of whole quads: a token's `top` rows are under way together.
// Every entry's sum keeps its order.  (64 -> 34 us for 2,048 tokens, 6 rows of 4,096.)
__device__ __forceinline__ float4 quad_of(const void* p, size_t i, int dtype) {
    if (dtype == MLS_BF16) {
        const uint2 raw = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p + i);
        const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
        const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
        return make_float4(lo.x, lo.y, hi.x, hi.y);
    }
    return *reinterpret_cast<const float4*>((const float*)p + i);
}
__device__ __forceinline__ void add4(float4& a, float4 b) {
    a.x += b.x;
    a.y += b.y;
    a.z += b.z;
    a.w += b.w;
}
template <typename T>
__global__ void __launch_bounds__(256)
expert_combine_quads_kernel(const float* __restrict__ per_slot, int top, const void* __restrict__ shared,
                            int shared_dtype, int shared_parts, size_t shared_stride,
                            const int* __restrict__ idx, const float* __restrict__ weight, int n_real,
                            const T* __restrict__ h, const float* __restrict__ gate, int gate_stride,
                            T* __restrict__ delta, int d) {
    chain_release();
    chain_wait();
    const size_t t = blockIdx.y;
    const int c = 4 * (blockIdx.x * blockDim.x + threadIdx.x);
    if (c >= d) return;
    const int dt = sizeof(T) == 2 ? MLS_BF16 : MLS_F32;
    const size_t i = t * d + c;
    float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
    constexpr int AT_ONCE = 8;
    for (int j0 = 0; j0 < top; j0 += AT_ONCE) {
        float4 v[AT_ONCE];
        float share[AT_ONCE];
        bool own[AT_ONCE];                    // a choice past the experts that have weights: its input
#pragma unroll
        for (int x = 0; x < AT_ONCE; ++x) {
            const size_t slot = t * top + j0 + x;
            own[x] = false;
            if (j0 + x >= top) continue;
            own[x] = idx && idx[slot] >= n_real;
            if (own[x]) {
                share[x] = weight[slot];
                v[x] = quad_of(h, i, dt);
            } else {
                v[x] = __ldcs(reinterpret_cast<const float4*>(per_slot + slot * d + c));
            }
        }
#pragma unroll
        for (int x = 0; x < AT_ONCE; ++x) {
            if (j0 + x >= top) continue;
            if (own[x])
                s = make_float4(s.x + share[x] * v[x].x, s.y + share[x] * v[x].y, s.z + share[x] * v[x].z,
                                s.w + share[x] * v[x].w);
            else
                add4(s, v[x]);
        }
    }
    if (shared) {
        float4 v = quad_of(shared, i, shared_dtype);
#pragma unroll 4
        for (int k = 1; k < shared_parts; ++k) add4(v, quad_of(shared, i + k * shared_stride, MLS_F32));
        if (gate) {
            const float f = 1.0f + expf(-gate[t * gate_stride]);
            v = make_float4(over(v.x, f), over(v.y, f), over(v.z, f), over(v.w, f));
        }
        add4(s, v);
    }
    if (sizeof(T) == 2) *reinterpret_cast<uint2*>(delta + i) = pack_bf16x4(s);
    else *reinterpret_cast<float4*>(delta + i) = s;
}
}  // namespace

MLS_API int mls_expert_tile_rows() { return BM; }

MLS_API int mls_route_topk(const float* logits, int logit_stride, int n_tokens, int n_experts,
                           int top, int renorm, int mode, const float* correction,
                           float renorm_eps, int n_groups, int keep_groups, int* idx,
                           float* weight, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (top <= 0 || top > n_experts) return MLS_ERR_UNSUPPORTED;
    if (n_groups > 1 && (n_groups > MAX_GROUPS || n_experts % n_groups || keep_groups < 1 ||
                         keep_groups > n_groups || top > keep_groups * (n_experts / n_groups)))
        return MLS_ERR_UNSUPPORTED;
#define TOPK_GO(HELD)                                                                              \
    MLS_LAUNCH((route_topk_kernel<HELD>), dim3((n_tokens + 3) / 4), dim3(128), 0, stream, logits,  \
               logit_stride, n_tokens, n_experts, top, renorm, mode, correction, renorm_eps,       \
               n_groups, keep_groups, idx, weight)
    if (n_experts <= 64) TOPK_GO(2);
    else if (n_experts <= 256) TOPK_GO(8);
    else TOPK_GO(0);
#undef TOPK_GO
    return launch_status();
}

MLS_API int mls_route_sort(const int* idx, int n_slots, int n_experts, int n_real, int* order,
                           int* offsets,
                           int* tile_expert, int* tile_row0, int max_tiles, int* cursor,
                           cudaStream_t stream) {
    if (n_slots <= 0) return 0;
    MLS_LAUNCH((route_sort_kernel), dim3(1), dim3(1024),
               n_experts <= SORT_SHARED ? n_experts * sizeof(int) : 0, stream, idx, n_slots, n_experts,
               n_real, order, offsets, tile_expert, tile_row0, max_tiles, cursor);
    return launch_status();
}

// Whether the products of these operands run on the tensor cores.
MLS_API int mls_expert_takes_tc(int dtype, const void* a, const void* w, int K) {
    return takes_tc(dtype, a, w, K) ? 1 : 0;
}

// One of the experts' products over the sorted slots: N outputs of K inputs an expert.  `rows`:
// scratch of n_slots x K bfloat16 for the sorted rows where the product runs on the tensor cores
// (unused otherwise, and by the down product, whose rows are sorted).
template <int UNIT>
static int expert_product(const void* A, const void* W, void* out, int dtype, const int* order,
                          const int* offsets, const int* tile_expert, const int* tile_row0,
                          int max_tiles, const float* weight, int top, int scale, int n_slots,
                          int n_experts, int N, int K, void* rows, float alpha, float limit,
                          int* status, cudaStream_t stream) {
    if (max_tiles <= 0) return 0;
    if (takes_tc(dtype, A, W, K)) {
        if (UNIT != DOWN) {
            if (!rows) return MLS_ERR_UNSUPPORTED;
            const int rc = gather_tc(A, order, weight, top, scale, n_slots, K, rows, stream);
            if (rc) return rc;
        }
        return product_tc(UNIT, UNIT == DOWN ? A : rows, W, out, order, offsets, weight, scale,
                          n_slots, n_experts, N, K, alpha, limit, status, stream);
    }
    const dim3 grid((N + BN - 1) / BN, max_tiles);
    if (dtype == MLS_BF16)
        MLS_LAUNCH((expert_gemm_kernel<__nv_bfloat16, UNIT>), dim3(grid), dim3(256), 0, stream,
                   (const __nv_bfloat16*)A, (const __nv_bfloat16*)W, out, order, offsets,
                   tile_expert, tile_row0, weight, top, scale, N, K, alpha, limit);
    else
        MLS_LAUNCH((expert_gemm_kernel<float, UNIT>), dim3(grid), dim3(256), 0, stream,
                   (const float*)A, (const float*)W, out, order, offsets, tile_expert, tile_row0,
                   weight, top, scale, N, K, alpha, limit);
    return launch_status();
}

MLS_API int mls_expert_glu(const void* h, const void* w_gate_up, void* y, int dtype,
                           const int* order, const int* offsets, const int* tile_expert,
                           const int* tile_row0, int max_tiles, const float* weight, int top,
                           int scale_in, int n_slots, int n_experts, int F, int K, void* rows,
                           float alpha, float limit, int* status, cudaStream_t stream) {
    return expert_product<GATED>(h, w_gate_up, y, dtype, order, offsets, tile_expert, tile_row0,
                                 max_tiles, weight, top, scale_in, n_slots, n_experts, F, K, rows,
                                 alpha, limit, status, stream);
}

MLS_API int mls_expert_relu2(const void* h, const void* w_up, void* y, int dtype, const int* order,
                             const int* offsets, const int* tile_expert, const int* tile_row0,
                             int max_tiles, const float* weight, int top, int scale_in, int n_slots,
                             int n_experts, int F, int K, void* rows, int* status,
                             cudaStream_t stream) {
    return expert_product<RELU2>(h, w_up, y, dtype, order, offsets, tile_expert, tile_row0, max_tiles,
                                 weight, top, scale_in, n_slots, n_experts, F, K, rows, 0.f, 0.f,
                                 status, stream);
}

MLS_API int mls_expert_down(const void* y, const void* w_down, float* per_slot, int dtype,
                            const int* order, const int* offsets, const int* tile_expert,
                            const int* tile_row0, int max_tiles, const float* weight, int top,
                            int scale_out, int n_slots, int n_experts, int D, int F, int* status,
                            cudaStream_t stream) {
    return expert_product<DOWN>(y, w_down, per_slot, dtype, order, offsets, tile_expert, tile_row0,
                                max_tiles, weight, top, scale_out, n_slots, n_experts, D, F, nullptr,
                                0.f, 0.f, status, stream);
}

MLS_API int mls_expert_combine(const float* per_slot, int top, const void* shared,
                               int shared_dtype, int shared_parts, long long shared_stride,
                               const int* idx, const float* weight, int n_real,
                               const void* h, const float* gate, int gate_stride, void* delta,
                               int dtype, int n_tokens, int d, cudaStream_t stream) {
    if (n_tokens <= 0) return 0;
    if (shared_parts > 1 && shared_dtype != MLS_F32) return MLS_ERR_UNSUPPORTED;
    auto quads = [](const void* p, int bytes) { return reinterpret_cast<uintptr_t>(p) % bytes == 0; };
    const int act = dtype == MLS_BF16 ? 8 : 16;
    // (Few or narrow rows are one short wave either way, and the loop over single entries ends sooner: 8
    // tokens of 512 entries, 8 rows each, 1.56 us, 1.81 by quads; 2,048 of 64 1.88, 2.76; 64 of 512 1.56, 1.69; 33 of
    // 1,024 1.68, 1.79.  130 of 512 1.93, 1.87; 64 of 2,048, 4 rows, 2.18, 1.77; 2,048 of them 20.0, 11.4.)
    if (d >= 256 && (long long)n_tokens * d >= 65536 &&
        d % 4 == 0 && shared_stride % 4 == 0 && n_tokens <= 65535 && quads(per_slot, 16) && quads(h, act) &&
        quads(delta, act) && quads(shared, shared_dtype == MLS_BF16 ? 8 : 16)) {
        const int threads = d >= 1024 ? 256 : 64;
        const dim3 grid((d / 4 + threads - 1) / threads, n_tokens);
        if (dtype == MLS_BF16)
            MLS_LAUNCH((expert_combine_quads_kernel<__nv_bfloat16>), grid, dim3(threads), 0, stream, per_slot,
                       top, shared, shared_dtype, shared_parts, (size_t)shared_stride, idx, weight, n_real,
                       (const __nv_bfloat16*)h, gate, gate_stride, (__nv_bfloat16*)delta, d);
        else
            MLS_LAUNCH((expert_combine_quads_kernel<float>), grid, dim3(threads), 0, stream, per_slot, top,
                       shared, shared_dtype, shared_parts, (size_t)shared_stride, idx, weight, n_real,
                       (const float*)h, gate, gate_stride, (float*)delta, d);
        return launch_status();
    }
    const size_t n = (size_t)n_tokens * d;
    const size_t want = (n + 255) / 256;
    const int blocks = (int)(want < (size_t)(8 * sm_count()) ? want : 8 * sm_count());
    if (dtype == MLS_BF16)
        MLS_LAUNCH((expert_combine_kernel<__nv_bfloat16>), dim3(blocks), dim3(256), 0, stream,
                   per_slot, top, shared, shared_dtype, shared_parts, (size_t)shared_stride, idx,
                   weight, n_real, (const __nv_bfloat16*)h,
                   gate, gate_stride, (__nv_bfloat16*)delta, n, d);
    else
        MLS_LAUNCH((expert_combine_kernel<float>), dim3(blocks), dim3(256), 0, stream, per_slot,
                   top, shared, shared_dtype, shared_parts, (size_t)shared_stride, idx, weight, n_real,
                   (const float*)h, gate, gate_stride,
                   (float*)delta, n, d);
    return launch_status();
}
