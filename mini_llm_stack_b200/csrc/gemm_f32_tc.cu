// Float32 products of long rows on the 5th-generation tensor cores (gemm_f32.h says which):
// out[M, N] = A[M, K] * W[N, K]^T, both operands float32 (A may be bfloat16).
//
// Every operand is the sum of three bfloat16 (8 + 8 + 8 bits of the 24 that a float32 has; the
// second and third round what the ones before left), and of the nine products of such parts the
// six that reach 2^-24 of the whole are added up:
//
//     a w ~ a1 w1 + (a1 w2 + a2 w1) + (a2 w2 + a1 w3 + a3 w1)
//
// each exact, in float32 accumulators.  The tensor cores cut off what an addition cannot hold, so an
// accumulator takes 64 of K only, the small products first; the sums of 64 are added up in float32
// registers, rounded to nearest, over a group of K (a sixteenth of it, 128 at least), and the groups'
// sums in their turn.  That order depends on K alone: a row's bits are the same whatever rows it is
// computed with, and whether a CTA walks all of K or one group (few rows), whose sum it then leaves to
// gemm_f32_parts_kernel.  Distance from float64 (2-norm over 2-norm, normal values) against one chain of fmaf
// over K: 0.92e-7 / 4.1e-7 at 512, 1.04e-7 / 8.1e-7 at 2,048, 1.23e-7 / 16.2e-7 at 8,192.
// Float32 operands are multiplied by 2^16 before they are split (bf16_parts.cuh says why), and the sums by what takes
// that back out, which rounds nothing but what becomes smaller than float32's normal numbers (2^-149 at most).
// A sum that is not finite (an operand that is infinite, not a number or 2^112 and more, or a sum of 2^96 and more,
// 2^112 with bfloat16 rows)
// is computed again as that chain.
//
// The weights take the 128-row side of the instruction: tiles of 128 x 32 come by TMA, a thread a row
// splits them in registers and puts the parts into tensor memory, from where the instruction reads
// its first operand.  That leaves shared memory, which would bound the product (three parts of both
// operands: 145 bytes a cycle of 128), to the rows' parts, up to 160 rows a tile, which
// split_rows_kernel has written once per product.  What bounds it: with many rows, per block of 32 of K and
// 160 rows, 960 cycles of instructions beside 46 KB from L2 (345 us of 651 in the largest product below, alone)
// and the splitting of the weights (50 us), which share shared memory; the weights' way from memory with few.
// The instructions are issued by one elected thread of a warp whose loop is uniform: from a branch that a
// single lane takes each cost some 50 cycles to prepare, which bounded every size (851 us for 651, 431 for 235).
//
// Measured against FFMA (us): 2,048 x 16,384 x 2,048 2,460 -> 648 (212 TFLOP/s), 515 x 16,384 x 2,048 721 -> 213,
// 515 x 2,048 x 8,192 510 -> 115, 16 x 2,048 x 8,192 250 -> 25, 3 x 128,256 x 2,048 393 -> 250 (1.05 GB: 4.2 TB/s),
// 1 x 2,048 x 2,048 22.5 -> 10.5; eight groups of K instead of sixteen leave 16 x 64 x 4,096 at 11.3 instead of 7.9.
//
// Warp roles: 0 = TMA producer, 1 = tensor memory and instructions, 4..7 = splitting the weights (a
// quarter of the lanes each), 8..15 = sums (two warps a quarter, 16 columns in turn).  Every
// wait is bounded; one that runs out sets MLS_STATUS_TIMEOUT, and the kernel frees its tensor memory
// and returns.
#include "bf16_parts.cuh"
#include "common.cuh"
#include "gemm_f32.h"
#include "tcgen05.cuh"
#include "tma.cuh"
#include <map>
#include <mutex>
#include <tuple>

namespace {
using namespace mls_tc;
using namespace mls_tma;

constexpr int BK = 32, UMMA_K = 16;                   // of K: a block, an instruction
constexpr int W_BYTES = UMMA_M * BK * 4;              // a block of weights
constexpr int ROW_BYTES = BK * 2;                     // a row of a part's block
constexpr int THREADS = 512;
constexpr int SUM_WARPS = 8, SPLIT_WARPS = 4;
constexpr int W_COLS = 3 * BK / 2, W_BUFS = 4;        // tensor memory of a block's parts; such blocks
constexpr int GROUPS = 16, GROUP_MIN = 128;
constexpr float UP = 65536.f;                         // of float32 operands
constexpr int MAX_STAGES = 12, RING_BYTES = 200 * 1024;

struct TcParams {
    const void* A;
    const float* W;
    float* out;                    // [M, N], or the groups' sums [groups, M, N]
    int M, N, K, a_f32;
    int nt, m_tiles;               // rows of a tile, tiles of rows
    int blocks, group, groups;     // blocks of K, blocks of a group, groups
    int cut;                       // a unit is one group of a tile
    int parts;                     // of a row's values: three, or the one that a bfloat16 is
    float down;                    // takes the operands' UP out of a sum
    int stages, stage_bytes;
    int* status;
};

// Four entries of a row of A: 0: float32 at 16 bytes, 1: bfloat16 at 8 bytes, 2: either type anywhere.
template <int KIND>
__device__ __forceinline__ float4 quad_of_row(const TcParams& p, size_t i) {
    if (KIND == 0) return *reinterpret_cast<const float4*>((const float*)p.A + i);
    if (KIND == 1) {
        const uint2 raw = *reinterpret_cast<const uint2*>((const __nv_bfloat16*)p.A + i);
        return make_float4(__uint_as_float(raw.x << 16), __uint_as_float(raw.x & 0xffff0000u),
                           __uint_as_float(raw.y << 16), __uint_as_float(raw.y & 0xffff0000u));
    }
    const int type = p.a_f32 ? MLS_F32 : MLS_BF16;
    return make_float4(load_as_float(p.A, i, type), load_as_float(p.A, i + 1, type), load_as_float(p.A, i + 2, type),
                       load_as_float(p.A, i + 3, type));
}
// The outputs (m0 + x, n), x < ROWS, that `which` names as chains over k, handed to `store` (rows past the last: that
// one once more).  Sixteen of k of the weights' row are in registers, the next ones under way, and the rows' loads
// are asked for together; once none of the named outputs is a number any more they are done.  (515 x 2,048 x 2,048, 70 us:
// rows that are no numbers took 13.9 ms entry by entry and output by output, now 79 us; one infinite value a row 14.4 ms,
// now 0.72; one such row 281 us, now 72.  FFMA takes 140 us for all of them.)
template <int KIND, int ROWS, typename Store>
__device__ __forceinline__ void chains_of(const TcParams& p, int m0, unsigned which, int n, Store store) {
    const int quads = p.K / 4, last = p.M - 1 - m0;      // (K is a multiple of four, the weights' rows lie at 16 bytes)
    const float4* w = reinterpret_cast<const float4*>(p.W + (size_t)n * p.K);
    const size_t at = (size_t)m0 * p.K;
    float s[ROWS];
    float4 b[4], next[4];
#pragma unroll
    for (int x = 0; x < ROWS; ++x) s[x] = 0.f;
#pragma unroll
    for (int y = 0; y < 4; ++y) next[y] = w[min(y, quads - 1)];
#pragma unroll 1
    for (int q = 0; q < quads; q += 4) {
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            b[y] = next[y];
            next[y] = w[min(q + 4 + y, quads - 1)];
        }
#pragma unroll
        for (int y = 0; y < 4; ++y) {
            if (q + y >= quads) break;
            float4 a[ROWS];
#pragma unroll
            for (int x = 0; x < ROWS; ++x)
                a[x] = quad_of_row<KIND>(p, at + (size_t)min(x, last) * p.K + 4 * (q + y));
#pragma unroll
            for (int x = 0; x < ROWS; ++x) {
                s[x] = fmaf(a[x].x, b[y].x, s[x]);
                s[x] = fmaf(a[x].y, b[y].y, s[x]);
                s[x] = fmaf(a[x].z, b[y].z, s[x]);
                s[x] = fmaf(a[x].w, b[y].w, s[x]);
            }
        }
        unsigned left = 0;
#pragma unroll
        for (int x = 0; x < ROWS; ++x) left |= s[x] == s[x] ? 1u << x : 0u;
        if (!(left & which)) break;
    }
#pragma unroll
    for (int x = 0; x < ROWS; ++x)
        if (which >> x & 1u) store(x, s[x]);
}
template <int ROWS, typename Store>
__device__ __forceinline__ void chains(const TcParams& p, int m0, unsigned which, int n, Store store) {
    const uintptr_t a = reinterpret_cast<uintptr_t>(p.A);
    if (p.a_f32 && a % 16 == 0) chains_of<0, ROWS>(p, m0, which, n, store);
    else if (!p.a_f32 && a % 8 == 0) chains_of<1, ROWS>(p, m0, which, n, store);
    else chains_of<2, ROWS>(p, m0, which, n, store);
}
// Rows of 64 bytes with the 64-byte swizzle; 8-row groups are 512 bytes apart.
__device__ __forceinline__ uint64_t rows_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)((8 * ROW_BYTES) >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                            // SWIZZLE_64B
    return d;
}

// Unit i: a tile (tiles of rows fastest, so that a tile of weights leaves memory once), and of K the
// blocks [from, to).
struct Unit {
    int n0, m0, from, to, g;
};
__device__ __forceinline__ Unit unit_of(const TcParams& p, int i) {
    const int tile = p.cut ? i / p.groups : i, g = p.cut ? i - tile * p.groups : 0;
    const int n = tile / p.m_tiles;
    return {n * UMMA_M, (tile - n * p.m_tiles) * p.nt, p.cut ? g * p.group : 0,
            p.cut ? min((g + 1) * p.group, p.blocks) : p.blocks, g};
}

// NT: the most rows of a tile.
template <int NT>
__global__ void __launch_bounds__(THREADS, 1)
gemm_f32_tc_kernel(const __grid_constant__ TcParams p, const __grid_constant__ CUtensorMap rows_map,
                   const __grid_constant__ CUtensorMap w_map) {
    extern __shared__ uint8_t smem_raw[];
    constexpr int ACCS = NT > 32 ? 2 : 4;
    constexpr int COLS = 512;
    static_assert(ACCS * NT + W_BUFS * W_COLS <= COLS, "tensor memory");
    __shared__ __align__(8) uint64_t bars[2 * MAX_STAGES + 2 * W_BUFS + 2 * ACCS];
    __shared__ uint32_t tmem_slot_s;
    const uint32_t base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    const uint32_t bar0 = smem_u32(bars);
    auto full = [&](int s) { return bar0 + 8u * s; };
    auto empty = [&](int s) { return bar0 + 8u * (MAX_STAGES + s); };
    auto w_full = [&](int b) { return bar0 + 8u * (2 * MAX_STAGES + b); };
    auto w_empty = [&](int b) { return bar0 + 8u * (2 * MAX_STAGES + W_BUFS + b); };
    auto acc_full = [&](int a) { return bar0 + 8u * (2 * MAX_STAGES + 2 * W_BUFS + a); };
    auto acc_empty = [&](int a) { return bar0 + 8u * (2 * MAX_STAGES + 2 * W_BUFS + ACCS + a); };

    // (the warp's number from a shuffle: what follows from it alone may stay in uniform registers, from
    // which the instructions take their operands)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int b = 0; b < W_BUFS; ++b) {
            mbar_init(w_full(b), SPLIT_WARPS);
            mbar_init(w_empty(b), 1);
        }
        for (int a = 0; a < ACCS; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), SUM_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(&tmem_slot_s), COLS);
        chain_release();                 // (not before: see there)
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *reinterpret_cast<volatile uint32_t*>(&tmem_slot_s);
    const int units = (p.N + UMMA_M - 1) / UMMA_M * p.m_tiles * (p.cut ? p.groups : 1);
    bool timed_out = false;

    if (warp < 4) {
        if (NT > 32) fewer_registers<40>();
        if (warp == 0 && lane == 0) {
            // ------------------------------------------------------------- TMA producer
            const uint32_t bytes = W_BYTES + p.parts * p.nt * ROW_BYTES;
            // the first ring of weights, which no kernel writes, before the rows are there
            int ahead = 0;
            if ((int)blockIdx.x < units) {
                const Unit u = unit_of(p, blockIdx.x);
                ahead = min(p.stages, u.to - u.from);
                for (int s = 0; s < ahead; ++s) {
                    mbar_arrive_expect_tx(full(s), bytes);
                    tma_load_2d(base + s * p.stage_bytes, &w_map, (u.from + s) * BK, u.n0, full(s));
                }
            }
            chain_wait();
            int g = 0, slot = 0;
            uint32_t turn = 1;                            // parity of the wait for an empty stage
            for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x) {
                const Unit u = unit_of(p, i);
                for (int kb = u.from; kb < u.to; ++kb, ++g) {
                    const uint32_t at = base + slot * p.stage_bytes;
                    if (g >= ahead) {
                        if (!mbar_wait(empty(slot), turn)) {
                            timed_out = true;
                            break;
                        }
                        mbar_arrive_expect_tx(full(slot), bytes);
                        tma_load_2d(at, &w_map, kb * BK, u.n0, full(slot));
                    }
                    for (int x = 0; x < p.parts; ++x)
                        tma_load_2d(at + W_BYTES + x * p.nt * ROW_BYTES, &rows_map, kb * BK, x * p.M + u.m0,
                                    full(slot));
                    if (++slot == p.stages) slot = 0, turn ^= 1;
                }
            }
            // the copies under way land before the block's shared memory goes away
            for (int j = g > p.stages ? g - p.stages : 0; j < g; ++j)
                if (!mbar_wait(full(j % p.stages), (j / p.stages) & 1)) timed_out = true;
        } else if (warp == 1) {
            // ------------------------------------------------------------- instructions
            const uint32_t idesc = umma_idesc(p.nt);
            const uint32_t part = p.nt * ROW_BYTES;
            int g = 0, c = 0, slot = 0;
            uint32_t turn = 0;
            for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x) {
                const Unit u = unit_of(p, i);
                for (int kb = u.from; kb < u.to; kb += 2, ++c) {
                    const int acc = c % ACCS, count = min(2, u.to - kb);
                    const uint32_t d = tmem_base + acc * NT;
                    if (!mbar_wait_warp(acc_empty(acc), ((c / ACCS) & 1) ^ 1)) timed_out = true;
                    uint32_t w[2], rows[2];
                    int stage[2];
                    // part x of the weights times part y of the rows, of block b
                    auto product = [&](int b, int x, int y, uint32_t accumulate) {
#pragma unroll
                        for (int kk = 0; kk < BK / UMMA_K; ++kk)
                            umma_ts(d, w[b] + x * (BK / 2) + kk * (UMMA_K / 2),
                                    rows_desc(rows[b] + y * part + kk * UMMA_K * 2), idesc, kk ? 1u : accumulate);
                    };
#pragma unroll
                    for (int b = 0; b < 2; ++b) {
                        if (b >= count || timed_out) break;
                        if (!mbar_wait_warp(full(slot), turn) || !mbar_wait_warp(w_full(g % W_BUFS), (g / W_BUFS) & 1)) {
                            timed_out = true;
                            break;
                        }
                        tc_fence_after();
                        stage[b] = slot;
                        w[b] = tmem_base + ACCS * NT + g % W_BUFS * W_COLS;
                        rows[b] = base + slot * p.stage_bytes + W_BYTES;
                        if (elect_one()) {
                            if (p.parts == 3) {
                                product(b, 1, 1, b);
                                product(b, 0, 2, 1);
                                product(b, 2, 0, 1);
                                product(b, 0, 1, 1);
                            } else {
                                product(b, 2, 0, b);
                            }
                            product(b, 1, 0, 1);
                        }
                        ++g;
                        if (++slot == p.stages) slot = 0, turn ^= 1;
                    }
                    if (timed_out) break;
                    if (elect_one()) {
                        product(0, 0, 0, 1);
                        umma_commit(empty(stage[0]));
                        umma_commit(w_empty((g - count) % W_BUFS));
                        if (count == 2) {
                            product(1, 0, 0, 1);
                            umma_commit(empty(stage[1]));
                            umma_commit(w_empty((g - 1) % W_BUFS));
                        }
                        umma_commit(acc_full(acc));
                    }
                    __syncwarp();
                }
            }
        }
    } else if (warp < 8) {
        // ----------------------------------------------------------- splitting the weights
        if (NT > 32) fewer_registers<88>();
        const int row = (warp & 3) * 32 + lane;
        const uint32_t lanes = (uint32_t)((warp & 3) * 32) << 16;
        int g = 0, slot = 0;
        uint32_t turn = 0;
        for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x) {
            const Unit u = unit_of(p, i);
            for (int kb = u.from; kb < u.to; ++kb, ++g) {
                const int buf = g % W_BUFS;
                if (!mbar_wait_warp(w_empty(buf), ((g / W_BUFS) & 1) ^ 1) || !mbar_wait_warp(full(slot), turn)) {
                    timed_out = true;
                    break;
                }
                tc_fence_after();
                const uint32_t w = tmem_base + ACCS * NT + buf * W_COLS + lanes;
                const uint32_t src = base + slot * p.stage_bytes + row * (BK * 4);
                unsigned long long v[16];                 // two values each: all loads first
#pragma unroll
                for (int x = 0; x < 8; ++x)              // 16 bytes x of the row, where the swizzle put them
                    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(v[2 * x]), "=l"(v[2 * x + 1])
                                 : "r"(src + ((x ^ (row & 7)) << 4)) : "memory");
#pragma unroll
                for (int x = 0; x < 16; ++x) v[x] = both_times(v[x], UP);
#pragma unroll
                for (int h = 0; h < 2; ++h) {
#pragma unroll
                    for (int y = 0; y < 3; ++y) {
                        uint32_t two[8];
#pragma unroll
                        for (int x = 0; x < 8; ++x) two[x] = bf16_part(v[8 * h + x]);
                        tmem_st8(w + y * (BK / 2) + h * 8, two);
                    }
                }
                tmem_st_wait();
                tc_fence_before();
                __syncwarp();
                if (lane == 0) mbar_arrive(w_full(buf));
                if (++slot == p.stages) slot = 0, turn ^= 1;
            }
        }
    } else {
        // ---------------------------------------------------------------------------- sums
        if (NT > 32) more_registers<192>();
        constexpr int R = NT / 32;
        const int q = warp & 3, half = (warp >> 2) & 1;
        const uint32_t lanes = (uint32_t)(q * 32) << 16;
        chain_wait();
        int c = 0;
        for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x) {
            const Unit u = unit_of(p, i);
            const int n = u.n0 + q * 32 + lane;
            float sum[R][16], all[R][16];
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int x = 0; x < 16; ++x) sum[r][x] = all[r][x] = 0.f;
            for (int k0 = u.from; k0 < u.to && !timed_out; k0 += p.group) {
                const int k1 = min(k0 + p.group, u.to);
                for (int kb = k0; kb < k1; kb += 2, ++c) {
                    const int acc = c % ACCS;
                    if (!mbar_wait_warp(acc_full(acc), (c / ACCS) & 1)) {
                        timed_out = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t d = tmem_base + acc * NT + lanes + half * 16;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        if (half * 16 + 32 * r >= p.nt) break;
                        uint32_t v[16];
                        tmem_ld16(d + 32 * r, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int x = 0; x < 16; ++x) sum[r][x] += __uint_as_float(v[x]);
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_empty(acc));
                }
#pragma unroll
                for (int r = 0; r < R; ++r)
#pragma unroll
                    for (int x = 0; x < 16; ++x) {
                        all[r][x] += sum[r][x];
                        sum[r][x] = 0.f;
                    }
            }
            if (timed_out || n >= p.N) continue;
            float* out = p.out + ((size_t)u.g * p.M + u.m0) * p.N + n;
            const int rows = min(p.nt, p.M - u.m0);
            const float down = p.cut ? 1.f : p.down;
            float any = 0.f;                              // zero as long as all are numbers
#pragma unroll
            for (int r = 0; r < R; ++r)
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    const int m = half * 16 + 32 * r + x;
                    any = fmaf(all[r][x], 0.f, any);
                    if (m < rows) out[(size_t)m * p.N] = all[r][x] * down;
                }
            if (any == 0.f || p.cut) continue;
            // what has just been stored says which are not finite: eight rows at a time
#pragma unroll 1
            for (int m = half * 16; m < rows; m += m & 8 ? 24 : 8) {
                float* const at = out + (size_t)m * p.N;
                unsigned which = 0;
                for (int x = 0; x < 8 && m + x < rows; ++x)
                    if (!finite(at[(size_t)x * p.N])) which |= 1u << x;
                if (which)
                    chains<8>(p, u.m0 + m, which, n, [&](int x, float v) { at[(size_t)x * p.N] = v; });
            }
        }
    }
    if (timed_out && p.status) atomicOr(p.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, COLS);
}

// The groups' sums of a cut product, added up in the groups' order.
__global__ void __launch_bounds__(256)
gemm_f32_parts_kernel(const __grid_constant__ TcParams p, const float* __restrict__ parts, float* __restrict__ out) {
    chain_release();
    chain_wait();
    const size_t size = (size_t)p.M * p.N;
    const size_t i = (size_t)blockIdx.x * 256 + threadIdx.x;
    if (i >= size) return;
    float v[GROUPS];
#pragma unroll
    for (int g = 0; g < GROUPS; ++g) v[g] = g < p.groups ? parts[g * size + i] : 0.f;
    float s = 0.f;
#pragma unroll
    for (int g = 0; g < GROUPS; ++g)
        if (g < p.groups) s += v[g];
    if (finite(s)) s *= p.down;
    else chains<1>(p, (int)(i / p.N), 1u, (int)(i % p.N), [&](int, float v) { s = v; });
    out[i] = s;
}

// The three parts of a float32 matrix (the one of a bfloat16 one): [parts, M, width] bfloat16, zeros past K.
// Eight entries a thread.
template <typename T, bool VEC>
__global__ void __launch_bounds__(256)
split_rows_kernel(const T* __restrict__ A, int M, int K, int width, __nv_bfloat16* __restrict__ parts) {
    chain_release();
    chain_wait();
    const int per = width / 8;
    const long long i = (long long)blockIdx.x * 256 + threadIdx.x;
    if (i >= (long long)M * per) return;
    const int m = (int)(i / per), k = 8 * (int)(i - (long long)m * per);
    const T* src = A + (size_t)m * K + k;
    float v[8];
    if (VEC && sizeof(T) == 4 && k + 8 <= K) {
        const float4 lo = *reinterpret_cast<const float4*>(src), hi = *reinterpret_cast<const float4*>(src + 4);
        v[0] = lo.x, v[1] = lo.y, v[2] = lo.z, v[3] = lo.w, v[4] = hi.x, v[5] = hi.y, v[6] = hi.z, v[7] = hi.w;
    } else {
#pragma unroll
        for (int x = 0; x < 8; ++x) v[x] = k + x < K ? Elem<T>::load(src + x) : 0.f;
    }
    unsigned long long two[4];
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        two[x] = beside(__float_as_uint(v[2 * x]), __float_as_uint(v[2 * x + 1]));
        if (sizeof(T) == 4) two[x] = both_times(two[x], UP);
    }
    uint4* dst = reinterpret_cast<uint4*>(parts + (size_t)m * width + k);
    const size_t apart = (size_t)M * per;
#pragma unroll
    for (int y = 0; y < (sizeof(T) == 4 ? 3 : 1); ++y) {
        uint4 out;
        out.x = bf16_part(two[0]);
        out.y = bf16_part(two[1]);
        out.z = bf16_part(two[2]);
        out.w = bf16_part(two[3]);
        dst[y * apart] = out;
    }
}

// Tensor maps by what they describe, as the bfloat16 products keep theirs.
struct MapKey {
    const void* ptr;
    long long rows, k, row_bytes;
    int f32, box_rows;
    bool operator<(const MapKey& o) const {
        return std::tie(ptr, rows, k, row_bytes, f32, box_rows) <
               std::tie(o.ptr, o.rows, o.k, o.row_bytes, o.f32, o.box_rows);
    }
};
// Blocks of BK values: of a float32 matrix (128-byte rows and swizzle) or of a bfloat16 one (64).
bool operand_map(const void* ptr, bool f32, long long rows, long long k, long long row_bytes, int box_rows,
                 CUtensorMap* out) {
    static std::map<MapKey, CUtensorMap> maps;
    static std::mutex lock;
    std::lock_guard<std::mutex> guard(lock);
    const MapKey key{ptr, rows, k, row_bytes, f32, box_rows};
    auto it = maps.find(key);
    if (it == maps.end()) {
        if (maps.size() > 4096) maps.clear();
        EncodeTiledFn fn = encode_fn();
        if (!fn) return false;
        CUtensorMap m;
        cuuint64_t gdim[2] = {(cuuint64_t)k, (cuuint64_t)rows};
        cuuint64_t gstride[1] = {(cuuint64_t)row_bytes};
        cuuint32_t box[2] = {BK, (cuuint32_t)box_rows};
        cuuint32_t estr[2] = {1, 1};
        if (fn(&m, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2,
               const_cast<void*>(ptr), gdim, gstride, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
               f32 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_64B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
               CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
        it = maps.emplace(key, m).first;
    }
    *out = it->second;
    return true;
}

constexpr int NT_FEW = 32, NT_MANY = 160;

struct Cut {
    int nt, m_tiles, blocks, group, groups, cut;
};
// Rows of a tile, and whether K is cut into its groups: what a simple count of cycles finds shortest.  A block
// of K takes some 600 + 6 nt cycles (2,048 x 16,384 x 2,048 with tiles of 80, 96, 128 and 160 rows: 1,130,
// 1,180, 1,390 and 1,550); a cut product writes and reads its groups' sums and launches one kernel more.
Cut cut_of(int M, int N, int K) {
    Cut best{};
    const int blocks = (K + BK - 1) / BK;
    const int least = GROUP_MIN / BK, share = ((blocks + GROUPS - 1) / GROUPS + 1) & ~1;
    const int group = share > least ? share : least, groups = (blocks + group - 1) / group;
    const long long n_tiles = (N + UMMA_M - 1) / UMMA_M, sms = sm_count();
    double least_cycles = 0;
    for (int most = 16; most <= NT_MANY; most += 16) {
        const int m_tiles = (M + most - 1) / most;
        const int nt = ((M + m_tiles - 1) / m_tiles + 15) & ~15;
        const double block = 600 + 6.0 * nt;
        for (int cut = 0; cut <= (groups > 1 ? 1 : 0); ++cut) {
            const long long units = n_tiles * m_tiles * (cut ? groups : 1), rounds = (units + sms - 1) / sms;
            double cycles = rounds * (block * (cut ? group : blocks) + 6.0 * nt) + 2000;
            if (cut) cycles += 3000 + 8.0 * groups * M * N / 2500;
            if (!best.nt || cycles < least_cycles) {
                least_cycles = cycles;
                best = {nt, m_tiles, blocks, group, groups, cut};
            }
        }
    }
    return best;
}

bool rows_are_their_part(const void* A, int a_dtype, int K) {
    return a_dtype == MLS_BF16 && K % 8 == 0 && reinterpret_cast<uintptr_t>(A) % 16 == 0;
}
long long parts_floats(const void* A, int a_dtype, int M, int K) {
    if (rows_are_their_part(A, a_dtype, K)) return 0;
    const long long width = (K + BK - 1) / BK * BK;            // multiples of 16 bytes throughout
    return (a_dtype == MLS_F32 ? 3 : 1) * (long long)M * width / 2;
}

template <int NT>
int launch_nt(const TcParams& p, const CUtensorMap& rows_map, const CUtensorMap& w_map, cudaStream_t stream) {
    const int smem = p.stages * p.stage_bytes + 1024;
    static bool configured = false;
    if (!configured) {
        // (one limit for all rings: with each product's own, a thread with a smaller ring could lower what
        // another had just raised)
        const cudaError_t e = cudaFuncSetAttribute(gemm_f32_tc_kernel<NT>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize, RING_BYTES + 1024);
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    const long long units = (long long)(p.N + UMMA_M - 1) / UMMA_M * p.m_tiles * (p.cut ? p.groups : 1);
    const int grid = (int)(units < sm_count() ? units : sm_count());
    MLS_LAUNCH((gemm_f32_tc_kernel<NT>), dim3(grid), dim3(THREADS), smem, stream, p, rows_map, w_map);
    return launch_status();
}
}  // namespace

namespace mls_f32 {
bool takes_tc(int a_dtype, const float* W, int N, int K) {
    if (K % 4 || reinterpret_cast<uintptr_t>(W) % 16) return false;
    if (N <= SKINNY_N)
        return N >= FEWEST_N && K >= (a_dtype == MLS_BF16 ? TC_K : 2 * TC_K) && (long long)N * K >= FEWEST_SIZE;
    return K >= TC_K || (K >= TC_K / 4 && (long long)N * K >= TC_SIZE);
}

long long tc_scratch_floats(const void* A, int a_dtype, int M, int N, int K) {
    const Cut c = cut_of(M, N, K);
    return parts_floats(A, a_dtype, M, K) + (c.cut ? (long long)c.groups * M * N : 0);
}

int tc_launches(const void* A, int a_dtype, int M, int N, int K) {
    return 1 + (rows_are_their_part(A, a_dtype, K) ? 0 : 1) + cut_of(M, N, K).cut;
}

int product_tc(const void* A, int a_dtype, const float* W, float* out, int M, int N, int K, float* scratch,
               int* status, cudaStream_t stream) {
    const Cut c = cut_of(M, N, K);
    const bool direct = rows_are_their_part(A, a_dtype, K);
    const long long floats = parts_floats(A, a_dtype, M, K);
    if (!scratch && (floats || c.cut)) return MLS_ERR_UNSUPPORTED;
    const int width = (K + BK - 1) / BK * BK;
    if (!direct) {
        const long long threads = (long long)M * (width / 8);
        const dim3 grid((unsigned)((threads + 255) / 256));
        __nv_bfloat16* parts = reinterpret_cast<__nv_bfloat16*>(scratch);
        if (a_dtype == MLS_BF16)
            MLS_LAUNCH((split_rows_kernel<__nv_bfloat16, false>), grid, dim3(256), 0, stream,
                       (const __nv_bfloat16*)A, M, K, width, parts);
        else if (reinterpret_cast<uintptr_t>(A) % 16 == 0)
            MLS_LAUNCH((split_rows_kernel<float, true>), grid, dim3(256), 0, stream, (const float*)A, M, K, width,
                       parts);
        else
            MLS_LAUNCH((split_rows_kernel<float, false>), grid, dim3(256), 0, stream, (const float*)A, M, K, width,
                       parts);
    }
    TcParams p{};
    p.A = A, p.W = W, p.M = M, p.N = N, p.K = K, p.a_f32 = a_dtype == MLS_F32;
    p.nt = c.nt, p.m_tiles = c.m_tiles, p.blocks = c.blocks, p.group = c.group, p.groups = c.groups, p.cut = c.cut;
    p.parts = a_dtype == MLS_F32 ? 3 : 1;
    p.down = a_dtype == MLS_F32 ? 1.f / (UP * UP) : 1.f / UP;
    p.out = c.cut ? scratch + floats : out;
    p.stage_bytes = W_BYTES + p.parts * c.nt * ROW_BYTES;
    p.stages = RING_BYTES / p.stage_bytes < MAX_STAGES ? RING_BYTES / p.stage_bytes : MAX_STAGES;
    p.status = status;
    CUtensorMap rows_map, w_map;
    const bool maps = direct ? operand_map(A, false, M, K, 2LL * K, c.nt, &rows_map)
                             : operand_map(scratch, false, (long long)p.parts * M, width, 2LL * width, c.nt, &rows_map);
    if (!maps || !operand_map(W, true, N, K, 4LL * K, UMMA_M, &w_map)) return MLS_ERR_TENSOR_MAP;
    const int rc = c.nt <= NT_FEW ? launch_nt<NT_FEW>(p, rows_map, w_map, stream)
                                  : launch_nt<NT_MANY>(p, rows_map, w_map, stream);
    if (rc || !c.cut) return rc;
    const size_t size = (size_t)M * N;
    MLS_LAUNCH((gemm_f32_parts_kernel), dim3((unsigned)((size + 255) / 256)), dim3(256), 0, stream, p,
               (const float*)p.out, out);
    return launch_status();
}
}  // namespace mls_f32
