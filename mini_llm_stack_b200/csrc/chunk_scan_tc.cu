// The chunk-wise scans' two large products on the 5th-generation tensor cores (chunk_scan.cu says what they
// are): every chunk's U = sum_s (..) k_s v_s^T, and its outputs [P | q] x [v; S0].
//
// Float32 throughout as in gemm_f32_tc.cu: an operand is the sum of three bfloat16 (values held in bfloat16
// are their own), six products of such parts are taken, accumulators hold 32 (outputs) or 64 (U) of k,
// the small products first, and are added up in float32 registers.
//
// Both products are taken transposed: f on the 128-row side of the instruction, from tensor memory, tokens
// (or e) on the other, from shared memory.  A thread owns a column j of the state: it reads S0[.., j] or v[.., j]
// straight from memory, its warp's 32 columns side by side, splits them in registers and puts the parts into
// its lane of tensor memory; and it finds U[.., j] or o[.., j] there, whose stores are whole lines again.  No
// operand of the wide side passes through shared memory.  A group of four warps walks its 128 columns by itself:
// convert a block of k, multiply, add up; two or four groups an SM hide each other's waits.  (Updates whose values are
// not bfloat16 as they lie, with silu or float32, take 160 columns of tensor memory a group, 512 for two: one such block
// has an SM at a time, the next waits for its columns.)
//
// A value that is infinite or not a number: in v it counts as zero for the tokens before it (P is lower
// triangular, but 0 x inf is not 0), and outputs from its token on are computed again as chains of fmaf, as is
// every sum that is not finite.
//
// What bounds it: latencies.  Of a block's 34,000 cycles for outputs (32 heads of 128 x 256) 8,000 go to the tokens'
// rows (three rounds of loads that all blocks of a wave ask for together, 3,000 cycles each), 20,000 to six blocks
// of k (700 converting, 900 until the instructions are under way, 500 the next loads, 150 waiting, 500 the sums).
// Where a head's rows leave shared memory for one block an SM only (e > 128) that one has four groups.
//
// Measured against FFMA (2,048 tokens): outputs of 32 heads of 128 x 256 192 -> 87 us, updates 114 -> 49; mLSTM's, 4
// heads of 256 x 512, 97 -> 39 (69 with two groups a block) and 64 -> 27.  Loops of loads that ask for their type
// inside, and a call of the chain inside the unrolled stores, made both slower than FFMA (254 and 255 us).
#include "bf16_parts.cuh"
#include "chunk_common.cuh"
#include "tcgen05.cuh"
#include "tma.cuh"

namespace {
using namespace mls_chunk;
using namespace mls_tc;
using namespace mls_tma;

constexpr int BK = 32, UMMA_K = 16;                   // of k: a block, an instruction
constexpr int TILE = C * 128;                         // bytes of 64 rows of 64 bfloat16
constexpr int BLOCK_COLS = 3 * BK / 2;                // tensor memory of a block's parts

// Four entries x .. x + 3 of row r (a multiple of four) as parts into three tiles of 64 x 64, one after the
// other, in the 128-byte swizzle.
__device__ __forceinline__ void put_parts(uint8_t* tiles, int r, int x, float4 v) {
    uint8_t* at = tiles + r * 128 + (((x >> 3) ^ (r & 7)) << 4) + (x & 7) * 2;
#pragma unroll
    for (int y = 0; y < 3; ++y) {
        uint2 two;
        two.x = bf16_part_up(v.x, v.y);
        two.y = bf16_part_up(v.z, v.w);
        *reinterpret_cast<uint2*>(at + y * TILE) = two;
    }
}
// The tokens' rows of q or k (times their factors) as parts into tiles of 64 x 64, zeros past the chunk's
// tokens and the head's size.  The loads of four quads a thread are under way together; the type is asked
// outside of the loops: within, every load would be waited for before the next.
template <int THREADS>
__device__ __forceinline__ void fill_parts(uint8_t* tiles, int n_tiles, const Rows& r, int silu, const Where& w,
                                           size_t t0, int head, const float* factor) {
    const size_t at = t0 * r.row + r.off + (size_t)head * r.width;
    constexpr int AHEAD = 4;
    for (int u0 = threadIdx.x; u0 < n_tiles * C * 16; u0 += AHEAD * THREADS) {
        float4 v[AHEAD];
        auto place = [&](int y, int& tile, int& t, int& x) {        // of quad y: false where there is none
            const int u = u0 + y * THREADS;
            tile = u / (C * 16), t = (u / 16) % C, x = 4 * (u % 16);
            return tile < n_tiles;
        };
        int tile, t, x;
        if (r.dtype == MLS_BF16) {
            uint2 raw[AHEAD];
#pragma unroll
            for (int y = 0; y < AHEAD; ++y) {
                const bool there = place(y, tile, t, x) && t < w.n && 64 * tile + x < r.width;
                raw[y] = there ? *reinterpret_cast<const uint2*>((const __nv_bfloat16*)r.base + at +
                                                                 (size_t)t * r.row + 64 * tile + x)
                               : make_uint2(0u, 0u);
            }
#pragma unroll
            for (int y = 0; y < AHEAD; ++y) {
                const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[y].x));
                const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw[y].y));
                v[y] = make_float4(lo.x, lo.y, hi.x, hi.y);
            }
        } else {
#pragma unroll
            for (int y = 0; y < AHEAD; ++y) {
                const bool there = place(y, tile, t, x) && t < w.n && 64 * tile + x < r.width;
                v[y] = there ? *reinterpret_cast<const float4*>((const float*)r.base + at + (size_t)t * r.row +
                                                                64 * tile + x)
                             : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        }
        if (silu)
#pragma unroll
            for (int y = 0; y < AHEAD; ++y)
                v[y] = make_float4(silu1(v[y].x), silu1(v[y].y), silu1(v[y].z), silu1(v[y].w));
#pragma unroll
        for (int y = 0; y < AHEAD; ++y)
            if (place(y, tile, t, x))
                put_parts(tiles + tile * 3 * TILE, t, x, factor ? times(v[y], factor[t]) : v[y]);
    }
}
// 32 values of this thread's lane into tensor memory: as they are (bfloat16 already), or as their parts.
__device__ __forceinline__ void put_lane(uint32_t taddr, float (&v)[BK], bool whole) {
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int y = 0; y < 3; ++y) {
            if (y && whole) break;
            uint32_t two[8];
#pragma unroll
            for (int x = 0; x < 8; ++x) two[x] = bf16_part_up(v[16 * h + 2 * x], v[16 * h + 2 * x + 1]);
            tmem_st8(taddr + y * (BK / 2) + h * 8, two);
        }
}
__device__ __forceinline__ void group_sync(int id) {
    asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory");
}
__device__ __forceinline__ float load_silu(const Rows& r, int silu, size_t i) {
    const float v = load_as_float(r.base, i, r.dtype);
    return silu ? silu1(v) : v;
}

// Entries 0 .. n - 1 (of 32, zeros behind) of a column whose entries are `apart` from each other.
__device__ __forceinline__ void load_column(const float* p, size_t apart, int n, float (&v)[BK]) {
    if (n >= BK) {
#pragma unroll
        for (int x = 0; x < BK; ++x, p += apart) v[x] = *p;
    } else {
#pragma unroll
        for (int x = 0; x < BK; ++x, p += apart) v[x] = x < n ? *p : 0.f;
    }
}
__device__ __forceinline__ void load_column(const __nv_bfloat16* q, size_t apart, int n, float (&v)[BK]) {
    const unsigned short* p = reinterpret_cast<const unsigned short*>(q);
    unsigned short raw[BK];
    if (n >= BK) {
#pragma unroll
        for (int x = 0; x < BK; ++x, p += apart) raw[x] = *p;
    } else {
#pragma unroll
        for (int x = 0; x < BK; ++x, p += apart) raw[x] = x < n ? *p : 0;
    }
#pragma unroll
    for (int x = 0; x < BK; ++x) v[x] = __uint_as_float((uint32_t)raw[x] << 16);
}
// The column's entries of tokens 32 b .. of v (the type is asked outside of the loops: within, every load would
// be waited for before the next); the first token that is no number goes into `odd`, and counts as zero.
__device__ __forceinline__ void load_v(const Args& a, const Where& w, int head, int j, int b, float (&v)[BK],
                                       int& odd) {
    const size_t at = ((size_t)w.t0 + BK * b) * a.v.row + a.v.off + (size_t)head * a.v.width + j;
    if (a.v.dtype == MLS_BF16) load_column((const __nv_bfloat16*)a.v.base + at, a.v.row, w.n - BK * b, v);
    else load_column((const float*)a.v.base + at, a.v.row, w.n - BK * b, v);
    if (a.silu)
#pragma unroll
        for (int x = 0; x < BK; ++x) v[x] = silu1(v[x]);
    float any = 0.f;                                      // zero as long as all are numbers
#pragma unroll
    for (int x = 0; x < BK; ++x) any = fmaf(v[x], 0.f, any);
    if (any != 0.f) {
#pragma unroll
        for (int x = 0; x < BK; ++x)
            if (!finite(v[x])) {
                odd = min(odd, BK * b + x);
                v[x] = 0.f;
            }
    }
}

// ------------------------------------------------------------------------------- update
constexpr int AGAIN = 8;                              // outputs of a column that are taken as chains together

// U[i, j] = sum_s factor_s k_s[i] v_s[j] for rows i of [i0, i1) of column j as chains: those that are not finite, or all.
__device__ __noinline__ void updates_again(const Args& a, const Where w, int head, const Rows kr, int k_silu, size_t k_t0,
                                           const float* factor, float* U, int i0, int i1, int j, bool all) {
    const size_t v_at = (size_t)w.t0 * a.v.row + a.v.off + (size_t)head * a.v.width + j;
    const size_t k_at = k_t0 * kr.row + kr.off + (size_t)head * kr.width;
    bool none = false;                                   // a value or a factor is no number, and so is the whole column
#pragma unroll 8
    for (int t = 0; t < w.n; ++t) {
        const float x = load_silu(a.v, a.silu, v_at + (size_t)t * a.v.row);
        none |= x != x || factor[t] != factor[t];
    }
    for (; i0 < i1; i0 += AGAIN) {
        if (none) {
            for (int x = 0; x < AGAIN && i0 + x < i1; ++x) U[(size_t)(i0 + x) * a.f + j] = NAN;
            continue;
        }
        unsigned which = 0;
        for (int x = 0; x < AGAIN && i0 + x < i1; ++x)
            if (all || !finite(U[(size_t)(i0 + x) * a.f + j])) which |= 1u << x;
        if (!which) continue;
        float s[AGAIN];
#pragma unroll
        for (int x = 0; x < AGAIN; ++x) s[x] = 0.f;
#pragma unroll 2
        for (int t = 0; t < w.n; ++t) {
            const float v = load_silu(a.v, a.silu, v_at + (size_t)t * a.v.row), f = factor[t];
#pragma unroll
            for (int x = 0; x < AGAIN; ++x)
                s[x] = fmaf(load_silu(kr, k_silu, k_at + (size_t)t * kr.row + min(i0 + x, i1 - 1)) * f, v, s[x]);
        }
#pragma unroll
        for (int x = 0; x < AGAIN; ++x)
            if (which >> x & 1u) U[(size_t)(i0 + x) * a.f + j] = s[x];
    }
}

template <int MODE, int GROUPS>
__global__ void __launch_bounds__(128 * GROUPS, 2)
chunk_update_tc_kernel(const __grid_constant__ Args a, const Scratch s, const Part part, const int cols) {
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    constexpr int THREADS = 128 * GROUPS;
    extern __shared__ uint8_t smem_raw[];
    __shared__ float factor[C];
    __shared__ __align__(8) uint64_t bars[GROUPS];
    __shared__ uint32_t tmem_slot_s;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* tiles = smem_raw + (base - raw);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int group = warp >> 2;
    if (threadIdx.x == 0) {
        for (int g = 0; g < GROUPS; ++g) mbar_init(smem_u32(&bars[g]), 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_slot_s), cols);
        chain_release();                 // (not before: see there)
    }
    if (threadIdx.x < C)
        factor[threadIdx.x] = row_factor<MODE>(a, s.rows_k, w, head, threadIdx.x, w.n - 1 - (int)threadIdx.x);
    Rows kr = a.k;
    if (MODE == TOKEN_DECAY) kr = Rows{s.rows_k, MLS_F32, a.n_heads * a.e, 0, a.e};
    const int k_silu = MODE == TOKEN_DECAY ? 0 : a.silu;
    const size_t k_t0 = MODE == TOKEN_DECAY ? w.idx * C : (size_t)w.t0;
    // (past the last column: that one once more, and nothing stored)
    const int column = (blockIdx.x * GROUPS + group) * 128 + (warp & 3) * 32 + lane, j = min(column, a.f - 1);
    const bool mine = (blockIdx.x * GROUPS + group) * 128 < a.f;
    const int blocks = w.n > BK ? 2 : 1;
    int odd = C;
    __syncthreads();
    // factor_s k_s: rows of k, e side by side (MN-major), tiles of 64 of e
    const int e_tiles = (a.e + 63) / 64;
    fill_parts<THREADS>(tiles, e_tiles, kr, k_silu, w, k_t0, head, factor);
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
    const bool whole = a.v.dtype == MLS_BF16 && !a.silu;
    const int block_cols = whole ? BK / 2 : BLOCK_COLS;
    const uint32_t acc = tmem_base + group * (64 + 2 * block_cols), A = acc + 64;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t bar = smem_u32(&bars[group]);
    float* U = s.states + (w.idx * a.n_heads + head) * state_floats(MODE, a.e, a.f);
    bool timed_out = false;
    if (mine) {
#pragma unroll 1
        for (int b = 0; b < blocks; ++b) {
            float v[BK];
            load_v(a, w, head, j, b, v, odd);
            put_lane(A + b * block_cols + lanes, v, whole);
        }
        tmem_st_wait();
        tc_fence_before();
        group_sync(1 + group);
        for (int tile = 0; tile < e_tiles; ++tile) {
            if ((warp & 3) == 0) {
                tc_fence_after();
                if (elect_one()) {
                    constexpr uint32_t idesc = umma_idesc(64, 1);
                    uint32_t accumulate = 0;
                    // part x of v times part y of k; the first of the next kind divides what is there
                    auto product = [&](int x, int y, bool next_kind) {
                        for (int kk = 0; kk < blocks * (BK / UMMA_K); ++kk) {
                            const uint32_t v = A + (kk >> 1) * block_cols + x * (BK / 2) + (kk & 1) * (UMMA_K / 2);
                            const uint64_t k = umma_desc_mn(base + (tile * 3 + y) * TILE + kk * UMMA_K * 128, TILE);
                            if (next_kind && kk == 0) umma_ts_onto<PART_SHIFT>(acc, v, k, idesc);
                            else umma_ts(acc, v, k, idesc, accumulate);
                            accumulate = 1;
                        }
                    };
                    if (!whole) product(1, 1, false);
                    product(0, 2, false);
                    if (!whole) product(2, 0, false);
                    product(0, 1, true);
                    if (!whole) product(1, 0, false);
                    product(0, 0, true);
                    umma_commit(bar);
                }
                __syncwarp();
            }
            if (!timed_out && !mbar_wait(bar, tile & 1)) timed_out = true;
            tc_fence_after();
            float any = odd < C ? 1.f : 0.f;               // zero as long as all are numbers
            float* dst = U + (size_t)(64 * tile) * a.f + j;
            const int n = column < a.f ? min(a.e - 64 * tile, 64) : 0;
#pragma unroll
            for (int c0 = 0; c0 < 64; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(acc + lanes + c0, r);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x, dst += a.f) {
                    any = fmaf(__uint_as_float(r[x]), 0.f, any);
                    if (c0 + x < n) *dst = __uint_as_float(r[x]);
                }
            }
            tc_fence_before();
            if (any != 0.f)
                updates_again(a, w, head, kr, k_silu, k_t0, factor, U, 64 * tile, 64 * tile + n, j, odd < C);
            group_sync(1 + group);
        }
    }
    if (MODE == MLSTM && blockIdx.x == 0) {
        for (int i = threadIdx.x; i < a.e; i += THREADS) {
            float n = 0.f;
            const size_t at = k_t0 * kr.row + kr.off + (size_t)head * kr.width + i;
            if (kr.dtype == MLS_BF16) {
                const __nv_bfloat16* src = (const __nv_bfloat16*)kr.base + at;
#pragma unroll 16
                for (int t = 0; t < w.n; ++t) n += __bfloat162float(src[(size_t)t * kr.row]) * factor[t];
            } else {
                const float* src = (const float*)kr.base + at;
#pragma unroll 16
                for (int t = 0; t < w.n; ++t) n += src[(size_t)t * kr.row] * factor[t];
            }
            U[(size_t)a.e * a.f + i] = n;
        }
    }
    if (timed_out && a.status) atomicOr(a.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, cols);
}

// ------------------------------------------------------------------------------- output
// o_t[j] = factor_t sum_i q_t[i] S0[i, j] + sum_s P_ts v_s[j] for the tokens t of column j that are not finite, and those
// from `odd` on, as chains.  Where the state is not a number the outputs are none already.  (The whole of 2,048 tokens
// behind one that is no number, 32 heads of 128 x 256, 0.68 ms: 5.96 ms an output at a time, 1.08 now; mLSTM's 4 heads of
// 256 x 512, 0.24 ms: 4.37, now 1.08.)
__device__ __noinline__ void outputs_again(const Args& a, const Where w, int head, const Rows qr, int q_silu, size_t q_t0,
                                           const float* factor, const float* P, const float* S, int odd, int j,
                                           float* out, size_t apart) {
    bool none = false;
#pragma unroll 16
    for (int i = 0; i < a.e; ++i) {
        const float x = S[(size_t)i * a.f + j];
        none |= x != x;
    }
    if (none) return;
    const size_t v_at = (size_t)w.t0 * a.v.row + a.v.off + (size_t)head * a.v.width + j;
    const size_t q_at = q_t0 * qr.row + qr.off + (size_t)head * qr.width;
    for (int t0 = 0; t0 < w.n; t0 += AGAIN) {
        unsigned which = 0;
        for (int x = 0; x < AGAIN && t0 + x < w.n; ++x)
            if (t0 + x >= odd || !finite(out[(t0 + x) * apart])) which |= 1u << x;
        if (!which) continue;
        float o[AGAIN], f[AGAIN];
#pragma unroll
        for (int x = 0; x < AGAIN; ++x) o[x] = 0.f, f[x] = factor[min(t0 + x, w.n - 1)];
        for (int s = 0; s < min(t0 + AGAIN, w.n); ++s) {
            const float v = load_silu(a.v, a.silu, v_at + (size_t)s * a.v.row);
#pragma unroll
            for (int x = 0; x < AGAIN; ++x)
                if (s <= t0 + x) o[x] = fmaf(P[(t0 + x) * C + s], v, o[x]);
        }
#pragma unroll 2
        for (int i = 0; i < a.e; ++i) {
            const float z = S[(size_t)i * a.f + j];
#pragma unroll
            for (int x = 0; x < AGAIN; ++x)
                o[x] = fmaf(load_silu(qr, q_silu, q_at + (size_t)min(t0 + x, w.n - 1) * qr.row + i) * f[x], z, o[x]);
        }
#pragma unroll
        for (int x = 0; x < AGAIN; ++x)
            if (which >> x & 1u) out[(t0 + x) * apart] = o[x];
    }
}

template <int MODE, int GROUPS>
__global__ void __launch_bounds__(128 * GROUPS, GROUPS == 4 ? 1 : 2)
chunk_output_tc_kernel(const __grid_constant__ Args a, const Scratch s, const Part part) {
    chain_wait();
    Where w;
    const int head = blockIdx.y;
    if (!locate<false>(a, part, blockIdx.z, w)) return;
    constexpr int THREADS = 128 * GROUPS, COLS = 128 * GROUPS;    // (a group: 64 + 48 columns)
    extern __shared__ uint8_t smem_raw[];
    __shared__ float factor[C];
    __shared__ __align__(8) uint64_t bars[GROUPS];
    __shared__ uint32_t tmem_slot_s;
    const uint32_t raw = smem_u32(smem_raw), base = (raw + 1023u) & ~1023u;
    uint8_t* tiles = smem_raw + (base - raw);
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    const int group = warp >> 2;
    if (threadIdx.x == 0) {
        for (int g = 0; g < GROUPS; ++g) mbar_init(smem_u32(&bars[g]), 1);
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(smem_u32(&tmem_slot_s), COLS);
        chain_release();                 // (not before: see there)
    }
    if (threadIdx.x < C)
        factor[threadIdx.x] = row_factor<MODE>(a, s.rows_q, w, head, threadIdx.x, threadIdx.x + 1);
    Rows qr = a.q;
    if (MODE == TOKEN_DECAY) qr = Rows{s.rows_q, MLS_F32, a.n_heads * a.e, 0, a.e};
    const int q_silu = MODE == TOKEN_DECAY ? 0 : a.silu;
    const size_t q_t0 = MODE == TOKEN_DECAY ? w.idx * C : (size_t)w.t0;
    const Reader q(qr, q_silu, w, head, q_t0);
    const size_t unit = w.idx * a.n_heads + head;
    const float* S = s.states + unit * state_floats(MODE, a.e, a.f);
    const float* P = s.scores + unit * C * C;
    // (past the last column: that one once more, and nothing stored)
    const int column = (blockIdx.x * GROUPS + group) * 128 + (warp & 3) * 32 + lane, j = min(column, a.f - 1);
    const bool mine = (blockIdx.x * GROUPS + group) * 128 < a.f;
    const int s_blocks = (a.e + BK - 1) / BK, blocks = s_blocks + (w.n > BK ? 2 : 1);
    float v[BK];
    int odd = C;                                          // the first of the column's tokens that is no number
    auto load = [&](int b) {
        if (b >= s_blocks) {
            load_v(a, w, head, j, b - s_blocks, v, odd);
            return;
        }
        load_column(S + (size_t)b * BK * a.f + j, a.f, a.e - BK * b, v);
    };
    if (mine) load(0);
    // the tokens' rows of q and of P as parts, tiles of 64 of k: q first
    const int q_tiles = (a.e + 63) / 64;
    fill_parts<THREADS>(tiles, q_tiles, qr, q_silu, w, q_t0, head, nullptr);
    constexpr int AHEAD = C * 16 / THREADS < 4 ? C * 16 / THREADS : 4;
#pragma unroll
    for (int u0 = 0; u0 < C * 16; u0 += AHEAD * THREADS) {
        float4 p[AHEAD];
#pragma unroll
        for (int y = 0; y < AHEAD; ++y)
            p[y] = reinterpret_cast<const float4*>(P)[u0 + y * THREADS + threadIdx.x];
#pragma unroll
        for (int y = 0; y < AHEAD; ++y) {
            const int u = u0 + y * THREADS + threadIdx.x;
            put_parts(tiles + q_tiles * 3 * TILE, u / 16, 4 * (u % 16), p[y]);
        }
    }
    fence_proxy_async();
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
    const uint32_t acc = tmem_base + group * (64 + BLOCK_COLS), A = acc + 64;
    const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
    const uint32_t bar = smem_u32(&bars[group]);
    bool timed_out = false;
    if (mine) {
        float sum[C];
#pragma unroll
        for (int t = 0; t < C; ++t) sum[t] = 0.f;
        for (int b = 0; b < blocks; ++b) {
            const bool whole = b >= s_blocks && a.v.dtype == MLS_BF16 && !a.silu;
            put_lane(A + lanes, v, whole);
            tmem_st_wait();
            tc_fence_before();
            group_sync(1 + group);
            if ((warp & 3) == 0) {
                tc_fence_after();
                if (elect_one()) {
                    constexpr uint32_t idesc = umma_idesc(C);
                    const int k = b < s_blocks ? b : 2 * q_tiles + b - s_blocks;      // block of the rows' tiles
                    const uint32_t rows = base + (k >> 1) * 3 * TILE + (k & 1) * BK * 2;
                    // part x of the state or v times part y of the tokens' rows; the first of the next kind
                    // divides what is there
                    enum { FIRST, ONTO, NEXT_KIND };
                    auto product = [&](int x, int y, int how) {
#pragma unroll
                        for (int kk = 0; kk < BK / UMMA_K; ++kk) {
                            const uint32_t s = A + x * (BK / 2) + kk * (UMMA_K / 2);
                            const uint64_t r = umma_desc(rows + y * TILE + kk * UMMA_K * 2);
                            if (how == NEXT_KIND && kk == 0) umma_ts_onto<PART_SHIFT>(acc, s, r, idesc);
                            else umma_ts(acc, s, r, idesc, how != FIRST || kk ? 1u : 0u);
                        }
                    };
                    product(0, 2, FIRST);
                    if (!whole) {
                        product(1, 1, ONTO);
                        product(2, 0, ONTO);
                    }
                    product(0, 1, NEXT_KIND);
                    if (!whole) product(1, 0, ONTO);
                    product(0, 0, NEXT_KIND);
                    umma_commit(bar);
                }
                __syncwarp();
            }
            if (b + 1 < blocks) load(b + 1);
            if (!timed_out && !mbar_wait(bar, b & 1)) timed_out = true;
            tc_fence_after();
#pragma unroll
            for (int c0 = 0; c0 < C; c0 += 16) {
                uint32_t r[16];
                tmem_ld16(acc + lanes + c0, r);
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x) sum[c0 + x] += __uint_as_float(r[x]);
            }
            if (MODE != TOKEN_DECAY && b == s_blocks - 1)
#pragma unroll
                for (int t = 0; t < C; ++t) sum[t] *= factor[t];
        }
        float any = odd < C ? 1.f : 0.f;
        float* const out = a.out + ((size_t)w.t0 * a.n_heads + head) * a.f + j;
        const size_t apart = (size_t)a.n_heads * a.f;
        const int n = column < a.f ? w.n : 0;
        float* dst = out;
#pragma unroll
        for (int t = 0; t < C; ++t, dst += apart) {
            any = fmaf(sum[t], 0.f, any);
            if (t < n) *dst = sum[t];
        }
        if (any != 0.f && n > 0) outputs_again(a, w, head, qr, q_silu, q_t0, factor, P, S, odd, j, out, apart);
    }
    if (MODE == MLSTM && blockIdx.x == 0) {
        // den_t = max(|P_t . 1 + factor_t q_t . n|, exp(-m_t)) + 1e-6: THREADS / 64 threads a token
        constexpr int PER = THREADS / C;
        const int t = threadIdx.x / PER, x0 = threadIdx.x % PER;
        const float* n = S + (size_t)a.e * a.f;
        float p[4] = {0.f, 0.f, 0.f, 0.f}, d[4] = {0.f, 0.f, 0.f, 0.f};
        for (int x = 4 * x0; x < C; x += 4 * PER) {
            const float4 y = *reinterpret_cast<const float4*>(P + t * C + x);
            p[0] += y.x, p[1] += y.y, p[2] += y.z, p[3] += y.w;
        }
        for (int i0 = 4 * x0; i0 < a.e; i0 += 4 * PER * 4) {
            float4 y[4], z[4];
#pragma unroll
            for (int g = 0; g < 4; ++g)
                z[g] = i0 + 4 * PER * g < a.e ? *reinterpret_cast<const float4*>(n + i0 + 4 * PER * g)
                                              : make_float4(0.f, 0.f, 0.f, 0.f);
            q.template quads<4>([&](int g) { return make_int2(t, i0 + 4 * PER * g); }, y);
#pragma unroll
            for (int g = 0; g < 4; ++g) {
                d[0] = fmaf(y[g].x, z[g].x, d[0]), d[1] = fmaf(y[g].y, z[g].y, d[1]);
                d[2] = fmaf(y[g].z, z[g].z, d[2]), d[3] = fmaf(y[g].w, z[g].w, d[3]);
            }
        }
        float all = ((p[0] + p[1]) + (p[2] + p[3])) + factor[t] * ((d[0] + d[1]) + (d[2] + d[3]));
#pragma unroll
        for (int o = 1; o < PER; o <<= 1) all += __shfl_xor_sync(0xffffffffu, all, o);
        if (x0 == 0 && t < w.n) {
            float* den = a.den + (size_t)(w.t0 + t) * a.n_heads + head;
            *den = fmaxf(fabsf(all), *den) + 1e-6f;
        }
    }
    if (timed_out && a.status) atomicOr(a.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem_base, COLS);
}

template <typename Kernel>
int allow(Kernel kernel, int smem) {
    return (int)cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
}
template <int MODE, int GROUPS>
int launch_update(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    const int smem = (a.e + 63) / 64 * 3 * TILE + 1024;
    const int rc = allow(chunk_update_tc_kernel<MODE, GROUPS>, smem);
    if (rc) return rc;
    // a group's accumulator of 64 columns and its two blocks
    const bool whole = a.v.dtype == MLS_BF16 && !a.silu;
    const int cols = (whole ? 128 : 256) * GROUPS;
    const dim3 grid((a.f + 128 * GROUPS - 1) / (128 * GROUPS), a.n_heads, part.chunks);
    MLS_LAUNCH((chunk_update_tc_kernel<MODE, GROUPS>), grid, dim3(128 * GROUPS), smem, stream, a, s, part, cols);
    return launch_status();
}
template <int MODE, int GROUPS>
int launch_output(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    const int smem = ((a.e + 63) / 64 + 1) * 3 * TILE + 1024;
    const int rc = allow(chunk_output_tc_kernel<MODE, GROUPS>, smem);
    if (rc) return rc;
    const dim3 grid((a.f + 128 * GROUPS - 1) / (128 * GROUPS), a.n_heads, part.chunks);
    MLS_LAUNCH((chunk_output_tc_kernel<MODE, GROUPS>), grid, dim3(128 * GROUPS), smem, stream, a, s, part);
    return launch_status();
}
}  // namespace

namespace mls_chunk {
template <int MODE>
int update_tc(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    return a.f <= 128 ? launch_update<MODE, 1>(a, s, part, stream) : launch_update<MODE, 2>(a, s, part, stream);
}
template <int MODE>
int output_tc(const Args& a, const Scratch& s, const Part& part, cudaStream_t stream) {
    if (a.f > 256 && a.e > 128) return launch_output<MODE, 4>(a, s, part, stream);
    return a.f <= 128 ? launch_output<MODE, 1>(a, s, part, stream) : launch_output<MODE, 2>(a, s, part, stream);
}
template int update_tc<HEAD_DECAY>(const Args&, const Scratch&, const Part&, cudaStream_t);
template int update_tc<TOKEN_DECAY>(const Args&, const Scratch&, const Part&, cudaStream_t);
template int update_tc<MLSTM>(const Args&, const Scratch&, const Part&, cudaStream_t);
template int output_tc<HEAD_DECAY>(const Args&, const Scratch&, const Part&, cudaStream_t);
template int output_tc<TOKEN_DECAY>(const Args&, const Scratch&, const Part&, cudaStream_t);
template int output_tc<MLSTM>(const Args&, const Scratch&, const Part&, cudaStream_t);
}  // namespace mls_chunk
