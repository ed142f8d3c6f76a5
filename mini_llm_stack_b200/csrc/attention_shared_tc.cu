// Causal attention for prompts and portions on the 5th-generation tensor cores where one cached
// row a token is both key and value (attention over a latent), heads of 256 entries.
//
// The kernel of attention_tc.cu ends at heads of 128: two chains of 128 rows with scores and outputs
// of 256 columns do not fit tensor memory, nor two rings of keys and values shared memory.  Here a
// tile of keys is brought in once and read twice, as the K-major operand of S = Q K^T and as the
// MN-major one of O += P V, and one chain of 128 rows keeps two score buffers, so that the
// tensor cores work on step i + 2's scores and step i's outputs while the softmax takes step i + 1.
// Tiles of 96 keys: three of them fit beside Q (48 KB each and 64 KB).
//
// The running maximum that the weights are taken against may lag behind by up to 2^8, so the largest
// weights of a row are not 1 but any number, and one bfloat16 would round each of them: on peaked rows
// two to three times the error of kernels that rescale at every new maximum.  A weight is therefore
// two bfloat16, the number rounded and what that left (16 bits together), and O += P V twice the
// instructions.  Distance from float64, 700 tokens of 8 heads, the output's own rounding included, for scores
// of deviation 1, 2 and 5: 1.58e-3, 1.64e-3, 1.65e-3; with one bfloat16 a weight 1.93e-3, 1.95e-3, 1.96e-3;
// the mma.sync tiles 1.90e-3, 1.80e-3, 1.70e-3.
//
//   warp 0      brings the tiles in with TMA, one copy per page and 64-wide quarter (one per quarter
//               for a run of consecutive pages);
//   warp 1      issues the products (tcgen05.mma);
//   warps 2..5  softmax, one thread a row: read S, mask, exponentiate, write P over it as two bfloat16,
//               rescale O when the running maximum has grown by more than 2^8, store O at the end.
//
// Measured against the mma.sync tiles (attention_mma.cu) on 32 heads over one latent of 256, prompts
// of 682 and 1,366 tokens: 230 -> 82 us (70 with one bfloat16 a weight: a step's products then were
// 12.6 MFLOP and are 18.9 now, half as much again for 16 % of the time, so it is the softmax, one warp a
// scheduler, that most of a step waits for; at the measured 1.65 PFLOP/s the products of a step take
// about 3,100 cycles).
// A key or value that is not a number reaches the earlier tokens of its tile of 128 rows, and of a tile whose last
// page it lies in (0 x NaN), as in attention_tc.cu; requests share no page.
// Every wait is bounded and reports MLS_STATUS_TIMEOUT.
#include "common.cuh"
#include "tma.cuh"
#include "tcgen05.cuh"
#include <map>
#include <mutex>
#include <tuple>

#ifndef MLS_HEAD_DIM
#error "compile with -DMLS_HEAD_DIM=<head size>"
#endif

#if MLS_HEAD_DIM == 256
namespace {
using namespace mls_tma;
using namespace mls_tc;

constexpr int HD = 256;
constexpr int ROWS = 128;                        // rows of a CTA: (token, head) pairs
constexpr int BN = 96;                           // keys of a tile
constexpr int QUARTERS = HD / 64;
constexpr int QBLOCK = ROWS * 128;               // bytes of [128 rows][64 elements]
constexpr int KBLOCK = BN * 128;                 // bytes of [96 keys][64 elements]
constexpr int Q_BYTES = QUARTERS * QBLOCK, K_STAGE = QUARTERS * KBLOCK, STAGES = 3;
constexpr int THREADS = 64 + ROWS;
constexpr int TMEM_COLS = 512, COL_O = 256;      // S0 at 0, S1 at 128, O
constexpr float LOG2E = 1.4426950408889634f;
constexpr float RESCALE_STEP = 8.0f;             // log2: P stays below 2^8

constexpr int B_K_FULL = 0, B_K_EMPTY = STAGES, B_S_FULL = 2 * STAGES, B_P_FULL = B_S_FULL + 2,
              B_O_REST = B_P_FULL + 2, B_O_LAST = B_O_REST + 1, B_Q_FULL = B_O_LAST + 1,
              N_BARS = B_Q_FULL + 1;
constexpr int SMEM_BYTES = Q_BYTES + STAGES * K_STAGE + 8 * N_BARS + 16;

struct Params {
    const __nv_bfloat16* qkv;
    __nv_bfloat16* out;
    const int* block_table;
    const int* cu_q;
    const int* ctx_len;
    int max_blocks, n_req, n_heads, n_kv, group, block_size, window, chunk, small_only, share;
    float scale_log2;
    int* status;
    long long n_pages;
    const float* sink;                           // [H] or nullptr
    long long out_stride;
};

__device__ __forceinline__ float fast_exp2(float x) {
    float y;
    asm("ex2.approx.ftz.f32 %0, %1;\n" : "=f"(y) : "f"(x));
    return y;
}
#define MLS_STATUS_BAD_SMEM 16       // dynamic shared memory is not 1024-byte aligned

__global__ void __launch_bounds__(THREADS)
attention_shared_tc_kernel(const Params P, const __grid_constant__ CUtensorMap kmap,
                           const __grid_constant__ CUtensorMap kmap_wide) {
    chain_wait();
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t base = smem_u32(smem_raw);
    if (base & 1023u) {                          // the swizzled tiles need this alignment
        if (threadIdx.x == 0 && P.status) atomicOr(P.status, MLS_STATUS_BAD_SMEM);
        return;
    }
    const uint32_t q_smem = base, k_smem = base + Q_BYTES, bars = k_smem + STAGES * K_STAGE;
    auto bar = [&](int i) { return bars + 8u * i; };
    volatile uint32_t* tmem_slot =
        reinterpret_cast<volatile uint32_t*>(smem_raw + (bars - base) + 8 * N_BARS);

    // which request and which tile of rows of it; the last rows see the most keys and go first
    int r = 0, tile = blockIdx.y, q_len = 0, rows = 0;
    for (; r < P.n_req; ++r) {
        q_len = P.cu_q[r + 1] - P.cu_q[r];
        rows = q_len * P.group;
        const bool small = P.small_only && q_len * (P.group / P.share) <= 16;
        const int tiles = small ? 0 : (rows + ROWS - 1) / ROWS;
        if (tile < tiles) break;
        tile -= tiles;
    }
    if (r >= P.n_req) return;
    tile = (rows + ROWS - 1) / ROWS - 1 - tile;
    const int kvh = blockIdx.x;
    // (the warp's number from a shuffle: what follows from it alone may stay in uniform registers, from which the
    // instructions take their operands)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int tok0 = P.cu_q[r], pos0 = P.ctx_len[r] - q_len;
    const int row0 = tile * ROWS;
    const int hi = pos0 + (min(rows, row0 + ROWS) - 1) / P.group;
    const int lo = max(0, first_visible(pos0 + row0 / P.group, P.window, P.chunk));
    const int* table = P.block_table + (size_t)r * P.max_blocks;
    const int kbase0 = (lo / BN) * BN;           // (a multiple of the page size, which divides 96)
    const int steps = (hi - kbase0) / BN + 1;

    if (threadIdx.x == 0) {
        for (int s = 0; s < STAGES; ++s) {
            mbar_init(bar(B_K_FULL + s), 1);
            mbar_init(bar(B_K_EMPTY + s), 1);
        }
        for (int b = 0; b < 2; ++b) {
            mbar_init(bar(B_S_FULL + b), 1);
            mbar_init(bar(B_P_FULL + b), ROWS);
        }
        mbar_init(bar(B_O_REST), 1);
        mbar_init(bar(B_O_LAST), 1);
        mbar_init(bar(B_Q_FULL), ROWS);
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), TMEM_COLS);
        chain_release();                 // (not before: see there)
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;
    bool timed_out = false;

    if (warp == 0) {
        // -------------------------------------------------------------- TMA producer
        const int bs = P.block_size, ppt = BN / bs;
        const uint32_t page_bytes = bs * 128;
        int t = 0;
        for (; t < steps; ++t) {
            const int slot = t % STAGES;
            const uint32_t full = bar(B_K_FULL + slot), stage = k_smem + slot * K_STAGE;
            if (!mbar_wait_warp(bar(B_K_EMPTY + slot), ((t / STAGES) & 1) ^ 1)) {
                timed_out = true;
                break;
            }
            bool valid = false;
            int page = -1;
            if (lane < ppt) {
                const int j0 = kbase0 + t * BN + lane * bs;
                if (j0 <= hi && j0 + bs > lo) {
                    page = table[j0 / bs];
                    valid = page >= 0;
                }
            }
            const unsigned mask = __ballot_sync(0xffffffffu, valid);
            const unsigned all = (1u << ppt) - 1u;
            const int first = __shfl_sync(0xffffffffu, page, 0);
            if (mask == all && __all_sync(0xffffffffu, lane >= ppt || page == first + lane)) {
                // pages that follow one another in the pool: one wide copy per quarter
                if (lane == 0) mbar_arrive_expect_tx(full, K_STAGE);
                __syncwarp();
                if (lane < QUARTERS)
                    tma_load_2d(stage + lane * KBLOCK, &kmap_wide, lane * 64,
                                (int)((kvh * P.n_pages + first) * bs), full);
                continue;
            }
            if (mask != all) {
                // pages that are not keys of this request read as zeros
                for (int pi = 0; pi < ppt; ++pi) {
                    if ((mask >> pi) & 1u) continue;
                    for (int part = 0; part < QUARTERS; ++part) {
                        const uint32_t dst = stage + part * KBLOCK + pi * page_bytes;
                        for (uint32_t o = lane * 16; o < page_bytes; o += 512)
                            asm volatile("st.shared.v4.u32 [%0], {%1, %1, %1, %1};\n" ::"r"(dst + o),
                                         "r"(0u) : "memory");
                    }
                }
                fence_proxy_async();
            }
            __syncwarp();
            if (lane == 0) mbar_arrive_expect_tx(full, __popc(mask) * page_bytes * QUARTERS);
            __syncwarp();
            if (valid) {
                const int y = (int)((kvh * P.n_pages + page) * bs);
#pragma unroll
                for (int h = 0; h < QUARTERS; ++h)
                    tma_load_2d(stage + h * KBLOCK + lane * page_bytes, &kmap, h * 64, y, full);
            }
        }
        // the copies under way land before the block's shared memory goes away
        for (int j = t > STAGES ? t - STAGES : 0; j < t; ++j)
            if (!mbar_wait_warp(bar(B_K_FULL + j % STAGES), (j / STAGES) & 1)) timed_out = true;
    } else if (warp == 1) {
        // ---------------------------------------------------------------- MMA issue
        {
            constexpr uint32_t idesc_s = umma_idesc(BN, 0);
            constexpr uint32_t idesc_o = umma_idesc(HD, 1);
            // S = Q K^T for step i, into the buffer whose P the product of step i - 2 has read
            // (the tensor cores run the instructions in the order they were issued)
            auto issue_s = [&](int i) -> bool {
                const int slot = i % STAGES;
                if (!mbar_wait_warp(bar(B_K_FULL + slot), (i / STAGES) & 1)) return false;
                tc_fence_after();
                const uint32_t k_src = k_smem + slot * K_STAGE;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < HD / 16; ++kk)
                        umma(tmem + (i & 1) * 128, umma_desc(q_smem + (kk >> 2) * QBLOCK + (kk & 3) * 32),
                             umma_desc(k_src + (kk >> 2) * KBLOCK + (kk & 3) * 32), idesc_s, kk ? 1u : 0u);
                    umma_commit(bar(B_S_FULL + (i & 1)));
                }
                __syncwarp();
                return true;
            };
            if (!mbar_wait_warp(bar(B_Q_FULL), 0)) timed_out = true;
            for (int i = 0; i < min(steps, 2) && !timed_out; ++i)
                if (!issue_s(i)) timed_out = true;
            for (int i = 0; i < steps && !timed_out; ++i) {
                if (!mbar_wait_warp(bar(B_P_FULL + (i & 1)), (i >> 1) & 1)) {
                    timed_out = true;
                    break;
                }
                tc_fence_after();
                const uint32_t v_src = k_smem + (i % STAGES) * K_STAGE;
                if (elect_one()) {
#pragma unroll
                    for (int kk = 0; kk < 2 * (BN / 16); ++kk) // the weights' upper halves, then the rest
                        umma_ts(tmem + COL_O, tmem + (i & 1) * 128 + kk * 8,
                                umma_desc_mn(v_src + kk % (BN / 16) * 16 * 128, KBLOCK), idesc_o,
                                (i | kk) ? 1u : 0u);
                    umma_commit(bar(i + 1 < steps ? B_O_REST : B_O_LAST));   // O holds step i
                    umma_commit(bar(B_K_EMPTY + i % STAGES));  // the tile has been read both ways
                }
                __syncwarp();
                if (i + 2 < steps && !issue_s(i + 2)) timed_out = true;
            }
        }
    } else {
        // ------------------------------------------------- softmax, correction, epilogue
        const int quarter = warp & 3;                          // its lanes of tensor memory
        const int row_in = quarter * 32 + lane, row = row0 + row_in;
        const bool live = row < rows;
        const int ti = live ? row / P.group : 0, g = live ? row - ti * P.group : 0;
        {
            // this thread's row of Q into shared memory, in the operand layout
            const int row_w = (P.n_heads + 2 * P.n_kv) * HD;
            const uint4* src = reinterpret_cast<const uint4*>(
                P.qkv + (size_t)(tok0 + ti) * row_w + (size_t)(kvh * P.group + g) * HD);
#pragma unroll
            for (int c0 = 0; c0 < HD / 8; c0 += 16) {
                uint4 v[16];
#pragma unroll
                for (int i = 0; i < 16; ++i) v[i] = live ? src[c0 + i] : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
                for (int i = 0; i < 16; ++i) {
                    const int ch = c0 + i;
                    asm volatile("st.shared.v4.u32 [%0], {%1, %2, %3, %4};\n"
                                 ::"r"(q_smem + (ch >> 3) * QBLOCK + row_in * 128 + (((ch & 7) ^ (row_in & 7)) << 4)),
                                   "r"(v[i].x), "r"(v[i].y), "r"(v[i].z), "r"(v[i].w) : "memory");
                }
            }
            fence_proxy_async();
            mbar_arrive(bar(B_Q_FULL));
        }
        const int pos = live ? pos0 + ti : -1;
        const int lo_row = first_visible(pos, P.window, P.chunk);
        const uint32_t lane_base = (uint32_t)(quarter * 32) << 16;
        const uint32_t o_addr = tmem + lane_base + COL_O;
        float m_used = -INFINITY, l = 0.f;
        for (int i = 0; i < steps && !timed_out; ++i) {
            const int kbase = kbase0 + i * BN;
            const uint32_t s_addr = tmem + lane_base + (i & 1) * 128;
            if (!mbar_wait_warp(bar(B_S_FULL + (i & 1)), (i >> 1) & 1)) {
                timed_out = true;
                break;
            }
            tc_fence_after();
            float sc[BN];
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 16) {
                uint32_t a[16];
                tmem_ld16(s_addr + c0, a);
#pragma unroll
                for (int e = 0; e < 16; ++e) sc[c0 + e] = __uint_as_float(a[e]);
            }
            tmem_ld_wait();
            const bool masked = kbase + BN - 1 > pos || kbase < lo_row;
            if (__any_sync(0xffffffffu, masked)) {
#pragma unroll
                for (int e = 0; e < BN; ++e) {
                    const int jj = kbase + e;
                    if (jj > pos || jj < lo_row) sc[e] = -INFINITY;
                }
            }
            float mx[8];
#pragma unroll
            for (int e = 0; e < 8; ++e) mx[e] = sc[e];
#pragma unroll
            for (int e = 8; e < BN; ++e) mx[e & 7] = fmaxf(mx[e & 7], sc[e]);
            const float m_tile = fmaxf(fmaxf(fmaxf(mx[0], mx[1]), fmaxf(mx[2], mx[3])),
                                       fmaxf(fmaxf(mx[4], mx[5]), fmaxf(mx[6], mx[7]))) *
                                 P.scale_log2;    // the scale is positive
            const bool grow = m_tile > m_used + RESCALE_STEP || (m_used == -INFINITY && m_tile > m_used);
            if (__any_sync(0xffffffffu, grow)) {
                const float m_new = grow ? m_tile : m_used;
                const float cf = (grow && m_used != -INFINITY) ? fast_exp2(m_used - m_new) : 1.0f;
                if (i > 0) {
                    // O must be at rest: the product of the step before has to be done (that of the
                    // one before it is, this step's scores were issued behind it)
                    if (!mbar_wait_warp(bar(B_O_REST), (i - 1) & 1)) {
                        timed_out = true;
                        break;
                    }
                    tc_fence_after();
#pragma unroll 2
                    for (int c0 = 0; c0 < HD; c0 += 32) {
                        uint32_t v[16], w[16];
                        tmem_ld16(o_addr + c0, v);
                        tmem_ld16(o_addr + c0 + 16, w);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            v[e] = __float_as_uint(__uint_as_float(v[e]) * cf);
                            w[e] = __float_as_uint(__uint_as_float(w[e]) * cf);
                        }
                        tmem_st16(o_addr + c0, v);
                        tmem_st16(o_addr + c0 + 16, w);
                    }
                }
                l *= cf;
                m_used = m_new;
            }
            const float neg_m = m_used == -INFINITY ? 0.f : -m_used;
            float part[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
            for (int c0 = 0; c0 < BN; c0 += 32) {
                uint32_t pk[16], rest[16];
#pragma unroll
                for (int u = 0; u < 16; ++u) {
                    const float p0 = fast_exp2(fmaf(sc[c0 + 2 * u], P.scale_log2, neg_m));
                    const float p1 = fast_exp2(fmaf(sc[c0 + 2 * u + 1], P.scale_log2, neg_m));
                    part[u & 3] += p0 + p1;
                    __nv_bfloat162 h = __floats2bfloat162_rn(p0, p1);
                    pk[u] = *reinterpret_cast<uint32_t*>(&h);
                    h = __floats2bfloat162_rn(p0 - __low2float(h), p1 - __high2float(h));
                    rest[u] = *reinterpret_cast<uint32_t*>(&h);
                }
                tmem_st16(s_addr + c0 / 2, pk);
                tmem_st16(s_addr + (BN + c0) / 2, rest);
            }
            l += (part[0] + part[1]) + (part[2] + part[3]);
            tmem_st_wait();                      // P and a rescaled O are in place
            tc_fence_before();
            mbar_arrive(bar(B_P_FULL + (i & 1)));
        }
        // All products are done once the last one is (they run in order).  It has a barrier of its own:
        // behind this thread's last arrival two phases of O_REST could end before it looks, and a parity
        // cannot tell a phase from the one two further on.
        if (!timed_out && !mbar_wait_warp(bar(B_O_LAST), 0)) timed_out = true;
        tc_fence_after();
        if (P.sink && live && m_used != -INFINITY)
            l += exp2f(P.sink[kvh * P.group + g] * LOG2E - m_used);
        const float inv = l > 0.f ? 1.0f / l : 0.f;
        __nv_bfloat16* dst = P.out + (size_t)(tok0 + ti) * P.out_stride + (size_t)(kvh * P.group + g) * HD;
#pragma unroll 2
        for (int c0 = 0; c0 < HD; c0 += 32) {
            uint32_t v[16], w[16];
            tmem_ld16(o_addr + c0, v);
            tmem_ld16(o_addr + c0 + 16, w);
            tmem_ld_wait();
            if (live) {
                uint32_t o[16];
#pragma unroll
                for (int e = 0; e < 8; ++e) {
                    __nv_bfloat162 h = __floats2bfloat162_rn(__uint_as_float(v[2 * e]) * inv,
                                                             __uint_as_float(v[2 * e + 1]) * inv);
                    o[e] = *reinterpret_cast<uint32_t*>(&h);
                    h = __floats2bfloat162_rn(__uint_as_float(w[2 * e]) * inv,
                                              __uint_as_float(w[2 * e + 1]) * inv);
                    o[8 + e] = *reinterpret_cast<uint32_t*>(&h);
                }
#pragma unroll
                for (int e = 0; e < 16; e += 4)
                    *reinterpret_cast<uint4*>(dst + c0 + 2 * e) = make_uint4(o[e], o[e + 1], o[e + 2], o[e + 3]);
            }
        }
    }
    if (timed_out && (threadIdx.x & 31) == 0 && P.status) atomicOr(P.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem, TMEM_COLS);
}

struct MapKey {
    const void* ptr;
    long long rows;
    int box;
    bool operator<(const MapKey& o) const { return std::tie(ptr, rows, box) < std::tie(o.ptr, o.rows, o.box); }
};
bool pool_map(const void* pool, long long pool_rows, int box, CUtensorMap* out) {
    static std::map<MapKey, CUtensorMap> maps;
    static std::mutex lock;
    std::lock_guard<std::mutex> guard(lock);
    const MapKey key{pool, pool_rows, box};
    auto it = maps.find(key);
    if (it == maps.end()) {
        if (maps.size() > 4096) maps.clear();
        CUtensorMap m;
        if (!make_map_bf16_2d(&m, pool, HD, (uint64_t)pool_rows, (uint64_t)HD * 2, 64, box)) return false;
        it = maps.emplace(key, m).first;
    }
    *out = it->second;
    return true;
}
}  // namespace
#endif

// Whether a pool whose rows are keys and values runs here: heads of 256, pages of 8, 16 or 32 tokens
// (they divide a tile of 96; other pages take the mma.sync tiles).
MLS_API int mls_attention_shared_tc_takes(int block_size) {
#if MLS_HEAD_DIM == 256
    return block_size == 8 || block_size == 16 || block_size == 32;
#else
    return 0;
#endif
}

// Prompts and portions of a step whose keys are their values: n_tiles = number of tiles of 128 rows
// over the requests (those that the split kernel takes are left out when skip_small is set).
MLS_API int mls_attention_shared_tc(const void* qkv, void* out, const void* pool, const int* block_table,
                                    int max_blocks, const int* cu_q, const int* ctx_len, int n_req,
                                    int n_heads, int n_kv, int block_size, float scale, int window,
                                    int n_tiles, int skip_small, long long pool_pages, int* status,
                                    const float* sink, long long out_stride, int chunk, int share,
                                    cudaStream_t stream) {
#if MLS_HEAD_DIM == 256
    if (n_tiles <= 0 || n_req <= 0) return 0;
    if (n_heads % n_kv || share < 1 || !mls_attention_shared_tc_takes(block_size) || out_stride % 8 ||
        !(scale > 0.f) ||
        (reinterpret_cast<uintptr_t>(qkv) | reinterpret_cast<uintptr_t>(out) |
         reinterpret_cast<uintptr_t>(pool)) % 16)
        return MLS_ERR_UNSUPPORTED;
    static bool configured = false;
    if (!configured) {
        const cudaError_t e = cudaFuncSetAttribute(attention_shared_tc_kernel,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, SMEM_BYTES);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    CUtensorMap kmap, kmap_wide;
    const long long rows = pool_pages * n_kv * block_size;
    if (!pool_map(pool, rows, block_size, &kmap) || !pool_map(pool, rows, BN, &kmap_wide))
        return MLS_ERR_TENSOR_MAP;
    Params P;
    P.qkv = (const __nv_bfloat16*)qkv;
    P.out = (__nv_bfloat16*)out;
    P.block_table = block_table;
    P.cu_q = cu_q;
    P.ctx_len = ctx_len;
    P.max_blocks = max_blocks;
    P.n_req = n_req;
    P.n_heads = n_heads;
    P.n_kv = n_kv;
    P.group = n_heads / n_kv;
    P.block_size = block_size;
    P.window = window;
    P.chunk = window > 0 ? 0 : chunk;
    P.small_only = skip_small ? 1 : 0;
    P.share = share;
    P.scale_log2 = scale * LOG2E;
    P.status = status;
    P.n_pages = pool_pages;
    P.sink = sink;
    P.out_stride = out_stride;
    MLS_LAUNCH((attention_shared_tc_kernel), dim3(n_kv, n_tiles), dim3(THREADS), SMEM_BYTES, stream, P,
               kmap, kmap_wide);
    return launch_status();
#else
    return MLS_ERR_UNSUPPORTED;
#endif
}
