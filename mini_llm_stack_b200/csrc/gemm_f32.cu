// True 32-bit matrix product for the float32 path: out[M, N] = A[M, K] * W[N, K]^T.
// A may be held in bfloat16 (a router's input in a 16-bit run): its values are widened as
// they are loaded, the arithmetic is the same.
// Long rows of many columns go to the tensor cores (gemm_f32_tc.cu; mls_f32::takes_tc says which); here
// are the others.
//
// FFMA on CUDA cores, two products an instruction where they lie side by side (fma.rn.f32x2
// rounds each as fmaf does): no tensor cores, no TF32, no reduced-precision mode.
// Each output element is accumulated over k = 0 .. K-1 in that order, whatever M
// and N are, so a token's result does not depend on the batch it is computed in.
// Both operands are K-contiguous (the reference's nn.Linear layout [out, in],
// train/model.py:79-82,130-132).
#include "common.cuh"
#include "gemm_f32.h"

namespace {
using namespace mls_f32;
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

// Four neighbouring values of a row, at a multiple of four elements' bytes.
__device__ __forceinline__ float4 load4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 load4(const __nv_bfloat16* p) {
    const uint2 raw = *reinterpret_cast<const uint2*>(p);
    const float2 lo = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.x));
    const float2 hi = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&raw.y));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
}
// Entries k .. k + 3 of a row of K, zeros past its end; VEC: they can be read at once.
template <bool VEC, typename T>
__device__ __forceinline__ float4 fetch4(const T* row, int k, int K) {
    if (VEC) return k < K ? load4(row + k) : make_float4(0.f, 0.f, 0.f, 0.f);
    return make_float4(k < K ? Elem<T>::load(row + k) : 0.f, k + 1 < K ? Elem<T>::load(row + k + 1) : 0.f,
                       k + 2 < K ? Elem<T>::load(row + k + 2) : 0.f, k + 3 < K ? Elem<T>::load(row + k + 3) : 0.f);
}

// A tile of BM x BN outputs a block, TM x 8 a thread.  Bound by the FFMA pipe (74 TFLOP/s) where
// there are enough tiles, else by the latency of a block of k.  Four lanes read a row's 16 of K
// (a lane a row would touch 32 lines a load, which cost more than the arithmetic); the tile is
// laid out transposed, row r of entries 4q.. at column r ^ 8q, so that neither the stores nor the
// 16-byte loads of four rows meet a bank twice.  The blocks of k after next are under way
// in registers, and two tiles in shared memory leave one barrier a block.
// Measured against 64 x 64 tiles of 4 x 4 a thread, loaded element by element and behind two
// barriers: 515 x 16,384 x 2,048 1,513 -> 718 us (48 TFLOP/s), 515 x 2,048 x 8,192 910 -> 506,
// 2,048 x 16,384 x 2,048 5,289 -> 2,551 (54), 64 x 2,048 x 2,048 155 -> 64 (sizes that the tensor cores
// take now).  The same bits.
constexpr int BK = 16, KQ = BK / 4;

template <typename T, bool VEC, int BM, int BN, int TM, int BLOCKS>
__global__ void __launch_bounds__((BM / TM) * (BN / 8), BLOCKS)
gemm_f32_kernel(const T* __restrict__ A, const float* __restrict__ W, float* __restrict__ out, int M,
                int N, int K) {
    constexpr int THREADS = (BM / TM) * (BN / 8), TXS = BN / 8;
    constexpr int NA = BM * KQ / THREADS, NW = BN * KQ / THREADS;    // quads of K a thread brings in
    static_assert(NA * THREADS == BM * KQ && NW * THREADS == BN * KQ && BM % 32 == 0 && BN % 64 == 0, "tile");
    chain_release();
    chain_wait();
    __shared__ __align__(16) float As[2][BK][BM];
    __shared__ __align__(16) float Ws[2][BK][BN];
    const int tid = threadIdx.x;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = tid % TXS, ty = tid / TXS;
    f32x2 acc[TM][4];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) acc[i][j] = 0ull;
    float4 fa[2][NA], fw[2][NW];
    auto fetch = [&](int k0, int set) {
#pragma unroll
        for (int x = 0; x < NA; ++x) {
            const int u = tid + x * THREADS, r = m0 + u / KQ;
            fa[set][x] = r < M ? fetch4<VEC>(A + (size_t)r * K, k0 + 4 * (u % KQ), K)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int x = 0; x < NW; ++x) {
            const int u = tid + x * THREADS, r = n0 + u / KQ;
            fw[set][x] = r < N ? fetch4<VEC>(W + (size_t)r * K, k0 + 4 * (u % KQ), K)
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    auto put = [&](int b, int set) {
#pragma unroll
        for (int x = 0; x < NA; ++x) {
            const int u = tid + x * THREADS, q = u % KQ, r = (u / KQ) ^ (8 * q);
            As[b][4 * q][r] = fa[set][x].x;
            As[b][4 * q + 1][r] = fa[set][x].y;
            As[b][4 * q + 2][r] = fa[set][x].z;
            As[b][4 * q + 3][r] = fa[set][x].w;
        }
#pragma unroll
        for (int x = 0; x < NW; ++x) {
            const int u = tid + x * THREADS, q = u % KQ, r = (u / KQ) ^ (8 * q);
            Ws[b][4 * q][r] = fw[set][x].x;
            Ws[b][4 * q + 1][r] = fw[set][x].y;
            Ws[b][4 * q + 2][r] = fw[set][x].z;
            Ws[b][4 * q + 3][r] = fw[set][x].w;
        }
    };
    // a thread's rows (columns) are runs of four, half a tile apart where there are eight
    auto compute = [&](int b) {
#pragma unroll
        for (int kk = 0; kk < BK; ++kk) {
            const int turn = 8 * (kk >> 2);
            float a[TM];
#pragma unroll
            for (int i = 0; i < TM; i += 4)
                *reinterpret_cast<float4*>(&a[i]) =
                    *reinterpret_cast<const float4*>(&As[b][kk][((ty * 4) ^ turn) + (i >> 2) * (BM / 2)]);
            const int col = (tx * 4) ^ turn;
            const ulonglong2 w0 = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][col]);
            const ulonglong2 w1 = *reinterpret_cast<const ulonglong2*>(&Ws[b][kk][col + BN / 2]);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const f32x2 two = twice(a[i]);
                fma2(acc[i][0], two, w0.x);
                fma2(acc[i][1], two, w0.y);
                fma2(acc[i][2], two, w1.x);
                fma2(acc[i][3], two, w1.y);
            }
        }
    };
    const int blocks = (K + BK - 1) / BK;
    fetch(0, 0);
    if (blocks > 1) fetch(BK, 1);
    put(0, 0);
    __syncthreads();
    for (int i = 0; i < blocks; i += 2) {
        if (i + 2 < blocks) fetch((i + 2) * BK, 0);
        compute(0);
        if (i + 1 >= blocks) break;
        put(1, 1);
        __syncthreads();
        if (i + 3 < blocks) fetch((i + 3) * BK, 1);
        compute(1);
        if (i + 2 < blocks) {
            put(0, 0);
            __syncthreads();
        }
    }
    const bool whole = N % 4 == 0 && reinterpret_cast<uintptr_t>(out) % 16 == 0;
#pragma unroll
    for (int i = 0; i < TM; ++i) {
        const int m = m0 + ty * 4 + (i >> 2) * (BM / 2) + (i & 3);
        if (m >= M) continue;
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const int n = n0 + tx * 4 + h * (BN / 2);
            const float2 lo = halves(acc[i][2 * h]), hi = halves(acc[i][2 * h + 1]);
            float* dst = out + (size_t)m * N + n;
            if (whole && n < N) {
                *reinterpret_cast<float4*>(dst) = make_float4(lo.x, lo.y, hi.x, hi.y);
            } else {
                if (n < N) dst[0] = lo.x;
                if (n + 1 < N) dst[1] = lo.y;
                if (n + 2 < N) dst[2] = hi.x;
                if (n + 3 < N) dst[3] = hi.y;
            }
        }
    }
}

// Up to FEW_M rows (decoding): what is read is W alone, and an output's sum is one chain over K
// (4 cycles a step).  Blocks of 64 of K come by asynchronous copies, STAGES of them under way.  With
// few columns a thread takes one output and a block 16 columns, so that every SM has a block; with
// many, whose reads of shared memory would bound it (426 us for 3 x 128,256 x 2,048), a thread
// takes four rows of a column and a block 64 columns.  Against the tiles of 32 x 64 above:
// 1 x 2,048 x 2,048 64 -> 17 us, 1 x 2,048 x 8,192 245 -> 55, 8 x 128,256 x 2,048 428 -> 391 (sizes that
// the tensor cores take now).  Rows of whole 16-byte pieces; the same bits.
constexpr int FEW_M = 8, FEW_K = 64, FEW_KP = FEW_K + 4;
template <int BN, int ROWS, int STAGES>
__global__ void __launch_bounds__(BN * (FEW_M / ROWS))
gemm_f32_few_kernel(const float* __restrict__ A, const float* __restrict__ W, float* __restrict__ out,
                    int M, int N, int K) {
    chain_release();
    extern __shared__ __align__(16) float stages[];          // [STAGES][BN + FEW_M][FEW_KP]
    constexpr int THREADS = BN * (FEW_M / ROWS), STAGE = (BN + FEW_M) * FEW_KP,
                  UNITS = (BN + FEW_M) * (FEW_K / 4);
    const int n0 = blockIdx.x * BN, n = threadIdx.x % BN, m0 = threadIdx.x / BN * ROWS;
    chain_wait();
    auto fetch = [&](int b) {                                // block b of K into its stage
        const int k0 = b * FEW_K;
        if (k0 < K) {
            float* st = stages + (b % STAGES) * STAGE;
#pragma unroll 4
            for (int u = threadIdx.x; u < UNITS; u += THREADS) {
                const int r = u / (FEW_K / 4), k = 4 * (u % (FEW_K / 4));
                const bool w = r < BN;
                const bool there = k0 + k < K && (w ? n0 + r < N : r - BN < M);
                const float* src = !there ? W : (w ? W + (size_t)(n0 + r) * K : A + (size_t)(r - BN) * K) + k0 + k;
                const uint32_t dst = (uint32_t)__cvta_generic_to_shared(st + r * FEW_KP + k);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n"
                             ::"r"(dst), "l"(src), "r"(there ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int b = 0; b < STAGES - 1; ++b) fetch(b);
    float acc[ROWS];
#pragma unroll
    for (int y = 0; y < ROWS; ++y) acc[y] = 0.f;
    const int blocks = (K + FEW_K - 1) / FEW_K;
    for (int b = 0; b < blocks; ++b) {
        asm volatile("cp.async.wait_group %0;\n" ::"n"(STAGES - 2) : "memory");
        __syncthreads();                                     // block b is there, block b - 1 is read
        fetch(b + STAGES - 1);
        const float* st = stages + (b % STAGES) * STAGE;
        const float* w = st + n * FEW_KP;
        const float* a = st + (BN + m0) * FEW_KP;
#pragma unroll
        for (int k = 0; k < FEW_K; k += 4) {
            const float4 y = load4(w + k);
#pragma unroll
            for (int r = 0; r < ROWS; ++r) {
                const float4 x = load4(a + r * FEW_KP + k);
                acc[r] = fmaf(x.x, y.x, acc[r]);
                acc[r] = fmaf(x.y, y.y, acc[r]);
                acc[r] = fmaf(x.z, y.z, acc[r]);
                acc[r] = fmaf(x.w, y.w, acc[r]);
            }
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
#pragma unroll
    for (int r = 0; r < ROWS; ++r)
        if (m0 + r < M && n0 + n < N) out[(size_t)(m0 + r) * N + n0 + n] = acc[r];
}

// Few output columns (a router's or a gate's scores: N <= SKINNY_N): the tile kernel above
// would leave all but a few SMs idle.  Here a warp owns SK_ROWS rows and COLS neighbouring
// columns; its lanes walk K four entries at a time with a stride of 128 (one entry at a time
// with a stride of 32 where rows are not whole 16-byte chunks), straight from memory: the warps
// of a block share rows, so all but the first read of a row meets L1.  The 32 partial sums are
// added by a fixed tree.  The order of the additions depends on K alone (never on M, on COLS or
// on the row's place), and which kernel runs depends on N alone, so a token's result still does
// not depend on its batch: many rows take eight or nine columns a warp (or four), fewer rows two, a
// decode step's one.  Measured against blocks of eight rows in shared memory, whose loads bounded it:
// 2,048 x 65 x 4,096 from bfloat16 rows 115 -> 45 us, 300 x 64 x 4,096 46 -> 16,
// 2,048 x 8 x 2,048 25 -> 8.
constexpr int SK_ROWS = 8;

// BY4: four entries of a row at a time, of both operands.
template <typename T, bool BY4, int COLS>
__global__ void __launch_bounds__(256)
gemm_f32_skinny_kernel(const T* __restrict__ A, const float* __restrict__ W, float* __restrict__ out,
                       int M, int N, int K) {
    chain_release();
    chain_wait();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int groups = (N + COLS - 1) / COLS;
    const int unit = blockIdx.x * 8 + warp;
    const int m0 = (unit / groups) * SK_ROWS, n0 = (unit % groups) * COLS;
    if (m0 >= M) return;
    float acc[COLS][SK_ROWS];
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r) acc[c][r] = 0.f;
    // rows and columns past the end read the last one; their sums are not stored
    const T* a_row[SK_ROWS];
#pragma unroll
    for (int r = 0; r < SK_ROWS; ++r) a_row[r] = A + (size_t)min(m0 + r, M - 1) * K;
    const float* w_row = W + (size_t)n0 * K;
    const int last = N - 1 - n0;
    if (BY4) {
#pragma unroll 2
        for (int k = lane * 4; k < K; k += 128) {
            float4 a[SK_ROWS];
#pragma unroll
            for (int r = 0; r < SK_ROWS; ++r) a[r] = load4(a_row[r] + k);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float4 w = load4(w_row + (size_t)min(c, last) * K + k);
#pragma unroll
                for (int r = 0; r < SK_ROWS; ++r) {
                    float s = acc[c][r];
                    s = fmaf(a[r].x, w.x, s);
                    s = fmaf(a[r].y, w.y, s);
                    s = fmaf(a[r].z, w.z, s);
                    acc[c][r] = fmaf(a[r].w, w.w, s);
                }
            }
        }
    } else {
        for (int k = lane; k < K; k += 32) {
            float a[SK_ROWS];
#pragma unroll
            for (int r = 0; r < SK_ROWS; ++r) a[r] = Elem<T>::load(a_row[r] + k);
#pragma unroll
            for (int c = 0; c < COLS; ++c) {
                const float w = w_row[(size_t)min(c, last) * K + k];
#pragma unroll
                for (int r = 0; r < SK_ROWS; ++r) acc[c][r] = fmaf(a[r], w, acc[c][r]);
            }
        }
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r) {
            const float s = warp_sum(acc[c][r]);
            if (lane == 0 && c <= last && m0 + r < M) out[(size_t)(m0 + r) * N + n0 + c] = s;
        }
}

// The same with a block's SK_ROWS rows of A in shared memory (all its warps' loads at once under way) and
// COLS columns a warp, with the loads of several rounds of W under way.  The same order of additions.
// One column a warp for the few rows of a decode step; four for many rows that cannot be read four
// entries at a time, where the kernel above has more than one wave of two columns a warp.
constexpr int SK_KC = 1024;
template <int COLS>
__global__ void __launch_bounds__(256)
gemm_f32_skinny_shared_kernel(const void* __restrict__ A, int a_dtype, const float* __restrict__ W,
                              float* __restrict__ out, int M, int N, int K, int by4) {
    chain_release();
    chain_wait();
    __shared__ __align__(16) float As[SK_ROWS][SK_KC];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int m0 = blockIdx.x * SK_ROWS;
    const int n0 = (blockIdx.y * 8 + warp) * COLS;
    float acc[COLS][SK_ROWS];
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r) acc[c][r] = 0.f;
    for (int k0 = 0; k0 < K; k0 += SK_KC) {
        const int kc = min(SK_KC, K - k0);
        __syncthreads();
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r)
            for (int k = threadIdx.x; k < kc; k += 256)
                As[r][k] = m0 + r < M ? load_as_float(A, (size_t)(m0 + r) * K + k0 + k, a_dtype) : 0.f;
        __syncthreads();
        if (n0 >= N) continue;
        if (by4) {
#pragma unroll 4
            for (int k = lane * 4; k < kc; k += 128) {
                float4 a[SK_ROWS];
#pragma unroll
                for (int r = 0; r < SK_ROWS; ++r) a[r] = *reinterpret_cast<const float4*>(&As[r][k]);
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    if (n0 + c >= N) break;
                    const float4 w = load4(W + (size_t)(n0 + c) * K + k0 + k);
#pragma unroll
                    for (int r = 0; r < SK_ROWS; ++r) {
                        float s = acc[c][r];
                        s = fmaf(a[r].x, w.x, s);
                        s = fmaf(a[r].y, w.y, s);
                        s = fmaf(a[r].z, w.z, s);
                        acc[c][r] = fmaf(a[r].w, w.w, s);
                    }
                }
            }
        } else {
            for (int k = lane; k < kc; k += 32) {
#pragma unroll
                for (int c = 0; c < COLS; ++c) {
                    if (n0 + c >= N) break;
                    const float w = W[(size_t)(n0 + c) * K + k0 + k];
#pragma unroll
                    for (int r = 0; r < SK_ROWS; ++r) acc[c][r] = fmaf(As[r][k], w, acc[c][r]);
                }
            }
        }
    }
#pragma unroll
    for (int c = 0; c < COLS; ++c)
#pragma unroll
        for (int r = 0; r < SK_ROWS; ++r) {
            const float s = warp_sum(acc[c][r]);
            if (lane == 0 && n0 + c < N && m0 + r < M) out[(size_t)(m0 + r) * N + n0 + c] = s;
        }
}

template <typename T, int COLS>
int skinny_shared(const T* A, const float* W, float* out, int M, int N, int K, bool by4, cudaStream_t stream) {
    MLS_LAUNCH((gemm_f32_skinny_shared_kernel<COLS>),
               dim3((M + SK_ROWS - 1) / SK_ROWS, (N + 8 * COLS - 1) / (8 * COLS)), dim3(256), 0, stream,
               (const void*)A, sizeof(T) == 2 ? MLS_BF16 : MLS_F32, W, out, M, N, K, by4 ? 1 : 0);
    return launch_status();
}

template <typename T>
int skinny(const T* A, const float* W, float* out, int M, int N, int K, bool vec_a, bool vec_w, cudaStream_t stream) {
    const int groups = (M + SK_ROWS - 1) / SK_ROWS;
#define SKINNY(BY4, C)                                                                             \
    do {                                                                                           \
        const long long warps = (long long)groups * ((N + C - 1) / C);                             \
        MLS_LAUNCH((gemm_f32_skinny_kernel<T, BY4, C>), dim3((unsigned)((warps + 7) / 8)),         \
                   dim3(256), 0, stream, A, W, out, M, N, K);                                      \
        return launch_status();                                                                    \
    } while (0)
    if (M < 64 || vec_a != vec_w)
        return M < 64 ? skinny_shared<T, 1>(A, W, out, M, N, K, vec_w, stream)
                      : skinny_shared<T, 4>(A, W, out, M, N, K, vec_w, stream);
    // Two columns a warp while those blocks are one wave (two an SM fit their registers): it is
    // then a warp's own chain of loads that counts, and a third of the registers lets more of them
    // be under way (512 x 64 x 4,096 from bfloat16 rows, after a flush of L2: 39 us with four
    // columns, 32 with eight, 23 with two; 128 x 128 x 2,048: 23, 19, 15).  Past that, A is read
    // once for eight columns (2,048 x 64 x 4,096: 102, 56, 62), or nine where that saves a group
    // (64 router outputs and a gate's column).  With float32 rows nine is the faster of the two
    // throughout (1,500 x 64 x 2,048: 45 us with eight, 36 with nine).
    const bool one_wave = (long long)groups * ((N + 1) / 2) <= 8LL * 2 * sm_count();
    const bool nine = (N + 8) / 9 < (N + 7) / 8;
    if (vec_a) {
        if (one_wave) SKINNY(true, 2);
        if constexpr (sizeof(T) == 2)
            if (!nine) SKINNY(true, 8);
        SKINNY(true, 9);
    }
    // Entry by entry the wide variants' loads bound them: they wait out fewer than eight warps an SM, and
    // float32 rows throughout, while shared memory serves four columns a warp (K = 1,023, wide / shared: float32
    // 1,500 x 33 50 / 25 us, 1,500 x 128 94 / 71; bfloat16 200 x 256 34 / 26, 1,500 x 64 25 / 49).  Two columns a
    // warp are one too many for one column (64 x 1 x 2,050 27 / 22 us) in float32.
    if (one_wave && (N > 1 || sizeof(T) == 2)) SKINNY(false, 2);
    if constexpr (sizeof(T) == 2)
        if ((long long)groups * ((N + 7) / 8) >= 8LL * sm_count()) {
            if (nine) SKINNY(false, 9);
            SKINNY(false, 8);
        }
    return skinny_shared<T, 4>(A, W, out, M, N, K, false, stream);
#undef SKINNY
}

template <typename T, bool VEC>
int tiled(const T* A, const float* W, float* out, int M, int N, int K, cudaStream_t stream) {
#define TILES(BM, BN, TM, BLOCKS)                                                                  \
    do {                                                                                           \
        MLS_LAUNCH((gemm_f32_kernel<T, VEC, BM, BN, TM, BLOCKS>),                                  \
                   dim3((N + BN - 1) / BN, (M + BM - 1) / BM), dim3((BM / TM) * (BN / 8)), 0,      \
                   stream, A, W, out, M, N, K);                                                    \
        return launch_status();                                                                    \
    } while (0)
    // 8 x 8 a thread reads the least from shared memory a product, but wants four blocks for every
    // SM; with fewer, smaller tiles keep more warps busy (us at 64 x 128 / 64 x 64 / 32 x 64:
    // 515 x 16,384 x 2,048 743 / 894 / -, 515 x 3,072 x 2,048 - / 176 / 196, 200 x 2,048 x 8,192
    // - / 312 / 301, 16 x 16,384 x 2,048 131 / 121 / 82)
    const long long sms = sm_count();
    auto tiles = [&](int bm, int bn) { return (long long)((M + bm - 1) / bm) * ((N + bn - 1) / bn); };
    if (M > 32 && tiles(64, 128) >= 4 * sms) TILES(64, 128, 8, 3);
    if (M > 32 && tiles(64, 64) * 2 >= 3 * sms) TILES(64, 64, 4, 4);
    TILES(32, 64, 4, 6);
#undef TILES
}

template <int BN, int ROWS, int STAGES>
int few_of(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t stream) {
    constexpr int smem = STAGES * (BN + FEW_M) * FEW_KP * (int)sizeof(float);
    static bool configured = false;
    if (!configured) {
        const int rc = (int)cudaFuncSetAttribute(gemm_f32_few_kernel<BN, ROWS, STAGES>,
                                                 cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
        if (rc) return rc;
        configured = true;
    }
    MLS_LAUNCH((gemm_f32_few_kernel<BN, ROWS, STAGES>), dim3((N + BN - 1) / BN), dim3(BN * (FEW_M / ROWS)),
               smem, stream, A, W, out, M, N, K);
    return launch_status();
}
int few(const float* A, const float* W, float* out, int M, int N, int K, cudaStream_t stream) {
    if (N >= 64 * 2 * sm_count()) return few_of<64, 4, 5>(A, W, out, M, N, K, stream);
    return few_of<16, 1, 8>(A, W, out, M, N, K, stream);
}

template <typename T>
int product(const T* A, int a_dtype, const float* W, float* out, int M, int N, int K, float* scratch, int* status,
            cudaStream_t stream) {
    const bool vec_a = K % 4 == 0 && reinterpret_cast<uintptr_t>(A) % (4 * sizeof(T)) == 0;
    const bool vec_w = K % 4 == 0 && reinterpret_cast<uintptr_t>(W) % 16 == 0;
    if (takes_tc(a_dtype, W, N, K)) return product_tc(A, a_dtype, W, out, M, N, K, scratch, status, stream);
    if (N <= SKINNY_N) return skinny(A, W, out, M, N, K, vec_a, vec_w, stream);
    if constexpr (sizeof(T) == 4)
        if (vec_w && vec_a && M <= FEW_M) return few(A, W, out, M, N, K, stream);
    if (vec_w && vec_a) return tiled<T, true>(A, W, out, M, N, K, stream);
    return tiled<T, false>(A, W, out, M, N, K, stream);
}
}  // namespace

// `scratch`: mls_gemm_f32_scratch_floats floats at a 16-byte address.
MLS_API int mls_gemm_f32(const void* A, int a_dtype, const float* W, float* out, int M, int N, int K,
                         float* scratch, int* status, cudaStream_t stream) {
    if (M <= 0 || N <= 0) return 0;
    if (a_dtype == MLS_F32)
        return product((const float*)A, a_dtype, W, out, M, N, K, scratch, status, stream);
    if (a_dtype == MLS_BF16)
        return product((const __nv_bfloat16*)A, a_dtype, W, out, M, N, K, scratch, status, stream);
    return MLS_ERR_UNSUPPORTED;
}

// Kernels that such a call launches.
MLS_API int mls_gemm_f32_launches(const void* A, int a_dtype, const float* W, int M, int N, int K) {
    if (M <= 0 || N <= 0) return 0;
    return takes_tc(a_dtype, W, N, K) ? tc_launches(A, a_dtype, M, N, K) : 1;
}

MLS_API long long mls_gemm_f32_scratch_floats(const void* A, int a_dtype, const float* W, int M, int N, int K) {
    return M > 0 && takes_tc(a_dtype, W, N, K) ? tc_scratch_floats(A, a_dtype, M, N, K) : 0;
}
