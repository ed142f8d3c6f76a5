// The experts' products of bfloat16 models on the 5th-generation tensor cores, expert by expert:
// for the sorted slots p of expert e (offsets[e] <= p < offsets[e + 1])
//
//   GATED   y[p, n] = unit(Wg[e] a_p, Wu[e] a_p)      W [E, 2N, K]: gate rows, then up rows
//   RELU2   y[p, n] = relu(Wu[e] a_p)^2               W [E, N, K]
//   DOWN    per_slot[order[p], n] = W[e] a_p          W [E, N, K], float32 out
//
// with a_p the sorted rows: for the first two what expert_gather_kernel wrote (a token's row,
// times the slot's weight where the design weighs inputs, rounded to bfloat16 once more), for
// DOWN the rows that the first product left.
//
// The weights take the 128-row side of the instruction and the expert's rows the other one, up
// to NT at a time and rounded up to 16 only: an expert of a prompt of 2,048 tokens has some 190
// rows (64 experts, 6 chosen), which tiles of 128 rows would fill to three quarters, and a
// decoded token's one row costs an instruction of 16.  What bounds it: every chosen expert's
// weights come from memory once (2.2 GB in that prompt, 0.34 ms at the copy bandwidth; its
// arithmetic takes 0.26 ms).  The units of work, (expert, 128 outputs, up to NT rows), are walked
// by one resident CTA an SM in that order, rows fastest, so that a tile of weights leaves memory
// once however many row tiles its expert has; the rows themselves stay in L2.  The gated unit
// has two accumulators, one for the gate's and one for the up rows of the same 128 outputs: one
// thread then holds both numbers of an output.
//
// Measured (2,048 tokens, 64 experts of 4,096 x 1,408, 6 chosen): gate / up 327 us and down 170 us
// where mma.sync tiles of 128 rows with synchronous loads took 2,173 and 1,209; 707 tokens, 32
// experts of 2,048 x 1,024 without a gate, 4 chosen: 41 + 37 us against 246 + 186; 16 tokens of
// the first: the whole feed-forward 357 us against 712 (1.8 GB of weights: 280 us).  The bits are
// those of the mma.sync tiles.
//
// Warp roles: 0 = TMA producer, 1 = tensor memory and instructions, 2..9 = epilogue (two warps a
// quarter of the lanes, taking 16 columns in turn).  Every output is its own sum over k
// ascending, whatever else is in the tile.  Every wait is bounded; one that runs out sets
// MLS_STATUS_TIMEOUT, and the kernel frees its tensor memory and returns.
#include "common.cuh"
#include "experts.h"
#include "tcgen05.cuh"
#include "tma.cuh"
#include <map>
#include <mutex>
#include <tuple>

namespace {
using namespace mls_tc;
using namespace mls_tma;
using namespace mls_experts;

constexpr int ROWS_W = UMMA_M;                       // outputs (weight rows) of a unit
constexpr int BK = 64, UMMA_K = 16;
constexpr int EPI_WARPS = 8;
constexpr int THREADS = 32 * (2 + EPI_WARPS);

template <int UNIT, int NT>
struct Plan {
    static constexpr int MATS = UNIT == GATED ? 2 : 1;             // accumulators of a unit
    static constexpr int ACCS = MATS * NT * 2 <= 512 ? 2 : 1;      // sets of them
    static constexpr int BOX = NT < 64 ? NT : 64;                  // rows of a copy
    static constexpr int A_BYTES = MATS * ROWS_W * BK * 2;
    static constexpr int STAGE = A_BYTES + NT * BK * 2;
    static constexpr int FIT = (200 * 1024) / STAGE;
    static constexpr int STAGES = FIT > 10 ? 10 : FIT;
    static constexpr int COLS_RAW = ACCS * MATS * NT;
    static constexpr int COLS = COLS_RAW < 32 ? 32 : COLS_RAW;     // NT is a power of two
    static constexpr int BARS = STAGES * STAGE;
    static constexpr int TMEM_SLOT = BARS + 8 * (2 * STAGES + 2 * ACCS);
    static constexpr int TABLE = TMEM_SLOT + 16;                   // [E + 1] ints follow
    static constexpr int FIXED = TABLE + 1024;                     // + alignment slack
};

struct TcParams {
    void* out;
    const int* order;
    const int* offsets;
    const float* weight;
    int n_experts, N, K, scale;
    float alpha, limit;
    int* status;
};

// Unit of work i: expert e, outputs from n0, rows [row0, row0 + rows).
struct Unit {
    int e, n0, row0, rows;
};
template <int NT>
__device__ __forceinline__ Unit unit_of(int i, int m_tiles, const int* start, int n_experts,
                                        const int* offsets) {
    const int q = i / m_tiles;
    int lo = 0, hi = n_experts;                       // start[lo] <= q < start[hi]
    while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (start[mid] <= q) lo = mid;
        else hi = mid;
    }
    const int tiles = start[lo + 1] - start[lo], j = i - start[lo] * m_tiles;
    const int m = j / tiles, t = j - m * tiles;
    const int p0 = offsets[lo], count = offsets[lo + 1] - p0;
    const int per = ((count + tiles - 1) / tiles + 15) & ~15;       // <= NT: even shares
    return {lo, m * ROWS_W, p0 + t * per, min(per, count - t * per)};
}

template <int UNIT, int NT>
__global__ void __launch_bounds__(THREADS, 1)
expert_tc_kernel(const TcParams p, const __grid_constant__ CUtensorMap rows_map,
                 const __grid_constant__ CUtensorMap w_map) {
    using L = Plan<UNIT, NT>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t raw = smem_u32(smem_raw);
    const uint32_t base = (raw + 1023u) & ~1023u;
    uint8_t* gbase = smem_raw + (base - raw);
    auto full = [&](int s) { return base + L::BARS + 8u * s; };
    auto empty = [&](int s) { return base + L::BARS + 8u * (L::STAGES + s); };
    auto acc_full = [&](int a) { return base + L::BARS + 8u * (2 * L::STAGES + a); };
    auto acc_empty = [&](int a) { return base + L::BARS + 8u * (2 * L::STAGES + L::ACCS + a); };
    volatile uint32_t* tmem_slot = reinterpret_cast<volatile uint32_t*>(gbase + L::TMEM_SLOT);
    int* start = reinterpret_cast<int*>(gbase + L::TABLE);

    // (the warp's number from a shuffle: what follows from it alone may stay in uniform registers, from which the
    // instructions take their operands)
    const int warp = __shfl_sync(0xffffffffu, threadIdx.x >> 5, 0), lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < L::STAGES; ++s) {
            mbar_init(full(s), 1);
            mbar_init(empty(s), 1);
        }
        for (int a = 0; a < L::ACCS; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), EPI_WARPS);
        }
        fence_barrier_init();
    }
    if (warp == 1) {
        tmem_alloc(smem_u32(const_cast<uint32_t*>(tmem_slot)), L::COLS);
        chain_release();                 // (not before: see there)
    }
    chain_wait();
    if (warp == 0) {
        // start[e]: row tiles of the experts before e.  A lane takes neighbouring experts, whose loads are
        // under way together (32 experts at a time were a chain of loads: 7.1 us for a decoded token of 600
        // experts of 256 x 128, 5.5 now).
        const int per = (p.n_experts + 31) / 32, e0 = min(lane * per, p.n_experts), e1 = min(e0 + per, p.n_experts);
        int sum = 0, at = e0 < e1 ? p.offsets[e0] : 0;
#pragma unroll 8
        for (int e = e0; e < e1; ++e) {
            const int next = p.offsets[e + 1];
            sum += (next - at + NT - 1) / NT;
            at = next;
        }
        int before = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int x = __shfl_up_sync(0xffffffffu, before, o);
            if (lane >= o) before += x;
        }
        if (lane == 31) start[p.n_experts] = before;
        before -= sum;
        at = e0 < e1 ? p.offsets[e0] : 0;
#pragma unroll 8
        for (int e = e0; e < e1; ++e) {
            const int next = p.offsets[e + 1];
            start[e] = before;
            before += (next - at + NT - 1) / NT;
            at = next;
        }
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    const int m_tiles = (p.N + ROWS_W - 1) / ROWS_W;
    const int units = start[p.n_experts] * m_tiles;
    const int kblocks = (p.K + BK - 1) / BK;
    bool timed_out = false;

    if (warp == 0) {
        // ----------------------------------------------------------------- TMA producer
        if (lane == 0) {
            int g = 0;
            for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x) {
                const Unit u = unit_of<NT>(i, m_tiles, start, p.n_experts, p.offsets);
                const int boxes = (u.rows + L::BOX - 1) / L::BOX;
                const uint32_t bytes = L::A_BYTES + boxes * (L::BOX * BK * 2);
                const int w_row = u.e * (L::MATS * p.N) + u.n0;
                for (int kb = 0; kb < kblocks; ++kb, ++g) {
                    const int slot = g % L::STAGES;
                    if (!mbar_wait(empty(slot), ((g / L::STAGES) & 1) ^ 1)) {
                        timed_out = true;
                        break;
                    }
                    const uint32_t a = base + slot * L::STAGE, b = a + L::A_BYTES;
                    mbar_arrive_expect_tx(full(slot), bytes);
                    tma_load_2d(a, &w_map, kb * BK, w_row, full(slot));
                    if (UNIT == GATED)
                        tma_load_2d(a + ROWS_W * BK * 2, &w_map, kb * BK, w_row + p.N, full(slot));
                    for (int x = 0; x < boxes; ++x)
                        tma_load_2d(b + x * (L::BOX * BK * 2), &rows_map, kb * BK,
                                    u.row0 + x * L::BOX, full(slot));
                }
            }
            // the copies under way land before the block's shared memory goes away
            for (int j = g > L::STAGES ? g - L::STAGES : 0; j < g; ++j)
                if (!mbar_wait(full(j % L::STAGES), (j / L::STAGES) & 1)) timed_out = true;
        }
    } else if (warp == 1) {
        // ---------------------------------------------------------------- instructions
        {
            int g = 0, it = 0;
            for (int i = blockIdx.x; i < units && !timed_out; i += gridDim.x, ++it) {
                const Unit u = unit_of<NT>(i, m_tiles, start, p.n_experts, p.offsets);
                const uint32_t idesc = umma_idesc((u.rows + 15) & ~15);
                const int acc = it % L::ACCS;
                if (!mbar_wait_warp(acc_empty(acc), ((it / L::ACCS) & 1) ^ 1)) {
                    timed_out = true;
                    break;
                }
                tc_fence_after();
                const uint32_t d = tmem_base + acc * (L::MATS * NT);
                for (int kb = 0; kb < kblocks; ++kb, ++g) {
                    const int slot = g % L::STAGES;
                    if (!mbar_wait_warp(full(slot), (g / L::STAGES) & 1)) {
                        timed_out = true;
                        break;
                    }
                    tc_fence_after();
                    const uint32_t a = base + slot * L::STAGE, b = a + L::A_BYTES;
                    if (elect_one()) {
#pragma unroll
                        for (int m = 0; m < L::MATS; ++m)
#pragma unroll
                            for (int kk = 0; kk < BK / UMMA_K; ++kk)
                                umma(d + m * NT, umma_desc(a + m * (ROWS_W * BK * 2) + kk * UMMA_K * 2),
                                     umma_desc(b + kk * UMMA_K * 2), idesc, (kb | kk) ? 1u : 0u);
                        umma_commit(empty(slot));
                    }
                    __syncwarp();
                }
                if (elect_one()) umma_commit(acc_full(acc));
                __syncwarp();
            }
        }
    } else {
        // -------------------------------------------------------------------- epilogue
        const int q = warp & 3, half = (warp - 2) >> 2;
        int it = 0;
        for (int i = blockIdx.x; i < units; i += gridDim.x, ++it) {
            const Unit u = unit_of<NT>(i, m_tiles, start, p.n_experts, p.offsets);
            const int acc = it % L::ACCS;
            const int n = u.n0 + q * 32 + lane;               // this thread's output
            const bool mine = n < p.N;
            if (!mbar_wait_warp(acc_full(acc), (it / L::ACCS) & 1)) {
                timed_out = true;
                break;
            }
            tc_fence_after();
            const uint32_t d = tmem_base + acc * (L::MATS * NT) + ((uint32_t)(q * 32) << 16);
#pragma unroll 1
            for (int c0 = half * 16; c0 < u.rows; c0 += 32) {
                uint32_t v[16], w[16];
                tmem_ld16(d + c0, v);
                if (UNIT == GATED) tmem_ld16(d + NT + c0, w);
                int slot = 0;
                float share = 1.f;
                if (UNIT == DOWN && lane < 16 && c0 + lane < u.rows) {
                    slot = p.order[u.row0 + c0 + lane];
                    if (p.scale) share = p.weight[slot];
                }
                tmem_ld_wait();
#pragma unroll
                for (int x = 0; x < 16; ++x) {
                    const float val = __uint_as_float(v[x]);
                    if (UNIT == DOWN) {
                        const int s = __shfl_sync(0xffffffffu, slot, x);
                        const float f = __shfl_sync(0xffffffffu, share, x);
                        if (mine && c0 + x < u.rows)
                            ((float*)p.out)[(size_t)s * p.N + n] = p.scale ? val * f : val;
                    } else if (mine && c0 + x < u.rows) {
                        const float r = UNIT == GATED
                                            ? gated_unit(val, __uint_as_float(w[x]), p.alpha, p.limit)
                                            : fmaxf(val, 0.f) * fmaxf(val, 0.f);
                        ((__nv_bfloat16*)p.out)[(size_t)(u.row0 + c0 + x) * p.N + n] =
                            __float2bfloat16_rn(r);
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty(acc));
        }
    }
    if (timed_out && p.status) atomicOr(p.status, MLS_STATUS_TIMEOUT);
    tc_fence_before();
    __syncthreads();
    if (warp == 1) tmem_dealloc(tmem_base, L::COLS);
}

// rows[p] = h[order[p] / top] (times weight[order[p]], rounded once more, with `scale`): 16 bytes
// a thread.
__global__ void __launch_bounds__(256)
expert_gather_kernel(const uint4* __restrict__ h, const int* __restrict__ order,
                     const float* __restrict__ weight, int top, int scale, int n_slots, int per_row,
                     uint4* __restrict__ rows) {
    chain_release();
    chain_wait();
    const int p = blockIdx.y;
    const int slot = order[p];
    const float share = scale ? weight[slot] : 1.f;
    const uint4* src = h + (size_t)(slot / top) * per_row;
    uint4* dst = rows + (size_t)p * per_row;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < per_row; i += gridDim.x * blockDim.x) {
        uint4 v = src[i];
        if (scale) {
            __nv_bfloat162* two = reinterpret_cast<__nv_bfloat162*>(&v);
#pragma unroll
            for (int x = 0; x < 4; ++x) {
                const float2 f = __bfloat1622float2(two[x]);
                two[x] = __floats2bfloat162_rn(f.x * share, f.y * share);
            }
        }
        dst[i] = v;
    }
}

// Tensor maps by what they describe, as the plain products keep theirs.
struct MapKey {
    const void* ptr;
    long long rows, k;
    int box_rows;
    bool operator<(const MapKey& o) const {
        return std::tie(ptr, rows, k, box_rows) < std::tie(o.ptr, o.rows, o.k, o.box_rows);
    }
};
bool operand_map(const void* ptr, long long rows, long long k, int box_rows, CUtensorMap* out) {
    static std::map<MapKey, CUtensorMap> maps;
    static std::mutex lock;
    std::lock_guard<std::mutex> guard(lock);
    const MapKey key{ptr, rows, k, box_rows};
    auto it = maps.find(key);
    if (it == maps.end()) {
        if (maps.size() > 4096) maps.clear();
        CUtensorMap m;
        if (!make_map_bf16_2d(&m, ptr, (uint64_t)k, (uint64_t)rows, (uint64_t)k * 2, BK, box_rows))
            return false;
        it = maps.emplace(key, m).first;
    }
    *out = it->second;
    return true;
}

template <int UNIT, int NT>
int launch_nt(const TcParams& p, const void* rows, const void* W, int n_slots, cudaStream_t stream) {
    using L = Plan<UNIT, NT>;
    const int smem = L::FIXED + 4 * (p.n_experts + 1);
    static bool configured = false;
    if (!configured) {
        // (one limit for all tables: with each product's own, a thread with a smaller table could lower what
        // another had just raised)
        const cudaError_t e = cudaFuncSetAttribute(expert_tc_kernel<UNIT, NT>,
                                                   cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                   L::FIXED + 4 * (TC_EXPERTS + 1));
        if (e != cudaSuccess) return (int)e;
        configured = true;
    }
    CUtensorMap rows_map, w_map;
    if (!operand_map(rows, n_slots, p.K, L::BOX, &rows_map) ||
        !operand_map(W, (long long)p.n_experts * L::MATS * p.N, p.K, ROWS_W, &w_map))
        return MLS_ERR_TENSOR_MAP;
    // the most units there can be: every expert's last row tile may be partly filled
    const long long tiles = (long long)(n_slots / NT) + (n_slots < p.n_experts ? n_slots : p.n_experts);
    const long long units = tiles * ((p.N + ROWS_W - 1) / ROWS_W);
    const int grid = (int)(units < sm_count() ? units : sm_count());
    MLS_LAUNCH((expert_tc_kernel<UNIT, NT>), dim3(grid), dim3(THREADS), smem, stream, p, rows_map,
               w_map);
    return launch_status();
}

// Rows of a tile (NT): the wider, the fewer times an expert's weights pass through shared memory;
// but the ring holds more stages where it is narrow (5 or 10 at 32, 4 or 6 at 128, 3 or 4 at 256),
// and at 256 the gated unit has one set of accumulators only, so that its epilogue is not hidden.
// The lines leave room for experts of twice the average before a second tile is needed at 32;
// from 96 on average a good part of the experts has more than 128 rows.
template <int UNIT>
int launch_unit(const TcParams& p, const void* rows, const void* W, int n_slots, int average,
                cudaStream_t stream) {
    if (average >= 96) return launch_nt<UNIT, 256>(p, rows, W, n_slots, stream);
    if (average >= 16) return launch_nt<UNIT, 128>(p, rows, W, n_slots, stream);
    return launch_nt<UNIT, 32>(p, rows, W, n_slots, stream);
}
}  // namespace

namespace mls_experts {
bool takes_tc(int dtype, const void* a, const void* w, int K) {
    return dtype == MLS_BF16 && K % 8 == 0 &&
           (reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(w)) % 16 == 0;
}

int product_tc(int unit, const void* rows, const void* W, void* out, const int* order,
               const int* offsets, const float* weight, int scale, int n_slots, int n_experts, int N,
               int K, float alpha, float limit, int* status, cudaStream_t stream) {
    if (n_slots <= 0 || N <= 0) return 0;
    const int average = n_slots / n_experts;
    // as many experts a launch as their table has room beside the stages
    for (int e0 = 0; e0 < n_experts; e0 += TC_EXPERTS) {
        const int n = n_experts - e0 < TC_EXPERTS ? n_experts - e0 : TC_EXPERTS;
        const TcParams p{out, order, offsets + e0, weight, n, N, K, scale, alpha, limit, status};
        const void* w = (const __nv_bfloat16*)W + (size_t)e0 * (unit == GATED ? 2 : 1) * N * K;
        const int rc = unit == GATED   ? launch_unit<GATED>(p, rows, w, n_slots, average, stream)
                       : unit == RELU2 ? launch_unit<RELU2>(p, rows, w, n_slots, average, stream)
                                       : launch_unit<DOWN>(p, rows, w, n_slots, average, stream);
        if (rc) return rc;
    }
    return 0;
}

int gather_tc(const void* h, const int* order, const float* weight, int top, int scale, int n_slots,
              int K, void* rows, cudaStream_t stream) {
    if (n_slots <= 0) return 0;
    const int per_row = K / 8;
    for (int p0 = 0; p0 < n_slots; p0 += 65535) {          // the grid's second dimension ends there
        const int n = n_slots - p0 < 65535 ? n_slots - p0 : 65535;
        MLS_LAUNCH((expert_gather_kernel), dim3((per_row + 1023) / 1024, n), dim3(256), 0, stream,
                   (const uint4*)h, order + p0, weight, top, scale, n, per_row,
                   (uint4*)rows + (size_t)p0 * per_row);
    }
    return launch_status();
}
}  // namespace mls_experts
