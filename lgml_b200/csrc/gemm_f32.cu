// 32-bit matrix product: C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]), float32 operands and results.  The order
// in which an output's products are added depends on K alone, whatever M, N and the tile it falls in, so a row's
// result does not depend on what else is in the batch.  It stands where mischief/lgml calls mul_mat with the f32
// flag (src/lgml.c:1811-1839).
//
// K >= 64: on the tensor cores, both operands in three bfloat16 parts that hold all their bits (below).  A chain of K dependent FMAs takes
// 4 cycles a step, and a K that is added up in segments can be shared out among warps.  Off 64 bits by (2-norm, chain of FMAs, here; random signs | one
// sign | one term in 16 | rows of one term):
//   K = 64    1.4e-7, 0.6e-7 | 1.1e-7, 0.5e-7 | 4.5e-8, 4.2e-8 | 2.5e-8, 2.5e-8
//   K = 256   2.9e-7, 0.8e-7 | 2.2e-7, 0.5e-7 | 7.5e-8, 6.0e-8 | 2.5e-8, 2.5e-8
//   K = 2048  8.1e-7, 1.1e-7 | 6.0e-7, 0.6e-7 | 2.1e-7, 0.9e-7 | 2.5e-8, 2.5e-8
//   K = 14336 2.1e-6, 2.1e-7 | 1.7e-6, 1.5e-7 | 5.4e-7, 2.0e-7 | 2.5e-8, 2.5e-8
//   * gemm_f32_few_kernel, up to 32 rows (or more of few features): warps stream W, each its segments of K.
//   * gemm_f32_many_kernel: tiles of 64 x 64.
// K < 64: every output sums its products in the order k = 0, 1, 2, ..., one chain of FMAs.
//   * gemm_f32_rows_kernel, one to four rows: a warp streams 8 or 16 rows of W through shared memory of its own.
//   * gemm_f32_tile_kernel, more rows: tiles of A and W by asynchronous copies, several blocks an SM.
//   * gemm_f32_ragged_kernel, more rows that do not all start on 16 bytes: tiles element by element.
// One B200, weights from HBM, launched one behind the other, microseconds, one chain of FMAs an output and now:
//   M, N, K:  4, 2048, 2048: 14.8 -> 10;  4, 2048, 5632: 31.2 -> 13.5;  4, 11264, 2048: 31 -> 22.4;  4, 32000, 2048: 59 -> 54 (4.9 TB/s);
//   32, 2048, 5632: 111 -> 38;  89, 2048, 5632: 160 -> 105;  89, 11264, 2048: 144 -> 177;  812, 11264, 2048: 883 -> 862;  2048, 32000, 2048: 5,879 -> 5,745.
// Two tf32 halves instead of the three parts (six tensor products a run for these eight) took 646 for 812 rows, 67 for 89 and 21 for 4 of 11,264, but
// held 23 bits: rows of one term were 8.6e-8 off, and one that selects a column did not give it exactly.

#include <type_traits>

#include "common.cuh"
#include "bf16_thirds.cuh"

LGML_DEFINE_LAST_ERROR(lgml_gemm_f32)

namespace {

__device__ __forceinline__ uint32_t smem_addr(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
// 16 bytes past L1 (what the kernel ahead wrote is read through L2); `bytes` of them from memory, zeros behind
__device__ __forceinline__ void cp_async_16(float *dst, const float *src, int bytes) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_addr(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// ---- few rows ------------------------------------------------------------------------------------
// A block is one warp: F features (lane % F) for up to MR = (32 / F) * MT rows of A, slot lane / F of the
// lanes taking MT of them.  A warp alone waits for its own copies only (no barrier between warps whose
// chains are all as long), and many small blocks put the stream of W on every SM.  A row of W is 128
// floats of a stage, one copy instruction of the warp; rows lie 132 floats apart, so that eight lanes'
// 16-byte reads of eight rows fall into all 32 banks.
constexpr int ROWS_BK = 128, ROWS_LD = ROWS_BK + 4;

template <int F, int MT> struct RowsShape {
    static constexpr int MR = 32 / F * MT;
    static constexpr int STAGES = F == 32 ? 3 : 4;
    static constexpr int STAGE_FLOATS = (F + MR) * ROWS_LD;
    static constexpr size_t SMEM = sizeof(float) * STAGES * STAGE_FLOATS;
};

template <int F, int MT, bool VEC, typename TO>
__global__ void __launch_bounds__(32) gemm_f32_rows_kernel(const float *__restrict__ A, const float *__restrict__ W, const float *__restrict__ bias,
                                                           TO *__restrict__ C, int M, int N, int K, int lda, int ldw, int ldc) {
    using S = RowsShape<F, MT>;
    constexpr int STAGES = S::STAGES;
    extern __shared__ __align__(16) float smem_f[];
    pdl_trigger();
    const int n0 = blockIdx.x * F, lane = threadIdx.x;
    const int n_kt = (K + ROWS_BK - 1) / ROWS_BK;
    auto stage = [&](int t) { return smem_f + (t % STAGES) * S::STAGE_FLOATS; };
    auto load_row = [&](float *dst, const float *row, bool there, int k0, bool act) {
        const int k = k0 + lane * 4;
        if constexpr (VEC) {
            const int bytes = there ? max(min(K - k, 4), 0) * 4 : 0;
            cp_async_16(dst + lane * 4, bytes > 0 ? row + k : W, bytes);
        } else {
#pragma unroll
            for (int i = 0; i < 4; ++i) {           // neighbouring lanes on neighbouring elements
                const int kk = i * 32 + lane;
                float v = 0.f;
                if (there && k0 + kk < K) v = act ? act_load(row + k0 + kk) : row[k0 + kk];
                dst[kk] = v;
            }
        }
    };
    auto load_w = [&](int t) {
#pragma unroll
        for (int r = 0; r < F; ++r) load_row(stage(t) + r * ROWS_LD, W + (size_t)min(n0 + r, N - 1) * ldw, n0 + r < N, t * ROWS_BK, false);
    };
    auto load_a = [&](int t) {
#pragma unroll
        for (int r = 0; r < S::MR; ++r)
            if (r < M) load_row(stage(t) + (F + r) * ROWS_LD, A + (size_t)r * lda, true, t * ROWS_BK, true);
    };
    // the weights of the first stages do not depend on the kernels ahead
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t)
        if (t < n_kt) load_w(t);
    pdl_wait();
#pragma unroll
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < n_kt) load_a(t);
        cp_async_commit();
    }
    const int f = lane % F, m_first = lane / F * MT;
    float acc[MT];
#pragma unroll
    for (int j = 0; j < MT; ++j) acc[j] = 0.f;
    for (int t = 0; t < n_kt; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncwarp();
        if (t + STAGES - 1 < n_kt) {
            load_w(t + STAGES - 1);
            load_a(t + STAGES - 1);
        }
        cp_async_commit();
        const float *ws = stage(t) + f * ROWS_LD;
        const float *as = stage(t) + (F + m_first) * ROWS_LD;
        // `ahead` times four k at a time, the next ones' reads under way while these ones' chain of FMAs runs (2,048 x 5,632, one to four
        // rows: 26 to 29 us, 29 to 33 with the reads where they are used; with eight rows a lane the chains alone fill the time)
        auto read = [&](int k, float4 &w, float4 (&a)[MT]) {
            w = *reinterpret_cast<const float4 *>(ws + k);
#pragma unroll
            for (int j = 0; j < MT; ++j) a[j] = *reinterpret_cast<const float4 *>(as + j * ROWS_LD + k);
        };
        auto add = [&](const float4 &w, const float4 (&a)[MT]) {
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] = fmaf(a[j].x, w.x, acc[j]);
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] = fmaf(a[j].y, w.y, acc[j]);
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] = fmaf(a[j].z, w.z, acc[j]);
#pragma unroll
            for (int j = 0; j < MT; ++j) acc[j] = fmaf(a[j].w, w.w, acc[j]);
        };
        {
            constexpr int AHEAD = 4, GROUPS = ROWS_BK / 4 / AHEAD;
            float4 w[2][AHEAD], a[2][AHEAD][MT];
#pragma unroll
            for (int u = 0; u < AHEAD; ++u) read(u * 4, w[0][u], a[0][u]);
#pragma unroll
            for (int g = 0; g < GROUPS; ++g) {
                if (g + 1 < GROUPS) {
#pragma unroll
                    for (int u = 0; u < AHEAD; ++u) read(((g + 1) * AHEAD + u) * 4, w[(g + 1) & 1][u], a[(g + 1) & 1][u]);
                }
#pragma unroll
                for (int u = 0; u < AHEAD; ++u) add(w[g & 1][u], a[g & 1][u]);
            }
        }
        __syncwarp();
    }
    const int n = n0 + f;
    if (n < N) {
        const float b = bias ? bias[n] : 0.f;
#pragma unroll
        for (int j = 0; j < MT; ++j) {
            const int m = m_first + j;
            if (m < M) C[(size_t)m * ldc + n] = from_f32<TO>(bias ? acc[j] + b : acc[j]);
        }
    }
}

// ---- tiles ---------------------------------------------------------------------------------------
// A tile of BM x BN outputs, TM x TN a thread, a warp 4 x 8 threads: rows ty + i * (BM / TM), columns
// tx + j * (BN / TN).  Both operands lie row by row in shared memory as they come (16-byte asynchronous
// copies, three stages in flight), rows 20 floats apart: the 16-byte reads of eight neighbouring rows
// fall into all 32 banks.  Several blocks an SM; for rows of 16-byte alignment.
template <int BM, int BN, int TM, int TN> struct TileShape {
    static constexpr int BK = 16, LD = BK + 4;
    static constexpr int TX = BN / TN, TY = BM / TM, THREADS = TX * TY;
    static constexpr int STAGES = 4;
    static constexpr int STAGE_FLOATS = (BM + BN) * LD;
    static constexpr size_t SMEM = sizeof(float) * STAGES * STAGE_FLOATS;
    static_assert(TX % 8 == 0 && TY % 4 == 0, "a warp is 4 x 8 threads");
    static_assert(BM * 4 % THREADS == 0 && BN * 4 % THREADS == 0, "whole copies per thread");
};

template <int BM, int BN, int TM, int TN, typename TO>
__global__ void __launch_bounds__(BM / TM *BN / TN) gemm_f32_tile_kernel(const float *__restrict__ A, const float *__restrict__ W,
                                                                         const float *__restrict__ bias, TO *__restrict__ C, int M, int N, int K,
                                                                         int lda, int ldw, int ldc, int tiles_m) {
    using S = TileShape<BM, BN, TM, TN>;
    constexpr int BK = S::BK, LD = S::LD, STAGES = S::STAGES, THREADS = S::THREADS;
    extern __shared__ __align__(16) float smem_f[];
    // row tiles fastest: the blocks that run at one time share a few column tiles of W, and A stays in L2
    const int m0 = (int)(blockIdx.x % tiles_m) * BM, n0 = (int)(blockIdx.x / tiles_m) * BN;
    const int n_kt = (K + BK - 1) / BK;
    auto stage = [&](int t) { return smem_f + (t % STAGES) * S::STAGE_FLOATS; };
    auto load = [&](float *dst, const float *src, int n_rows, int row0, int rows, int k0, int ld) {
#pragma unroll
        for (int c0 = 0; c0 < n_rows * (BK / 4); c0 += THREADS) {
            const int c = c0 + (int)threadIdx.x;
            const int r = c / (BK / 4), kk = (c % (BK / 4)) * 4;
            const int bytes = row0 + r < rows ? max(min(K - k0 - kk, 4), 0) * 4 : 0;
            cp_async_16(dst + r * LD + kk, bytes > 0 ? src + (size_t)(row0 + r) * ld + k0 + kk : src, bytes);
        }
    };
    auto load_w = [&](int t) { load(stage(t) + BM * LD, W, BN, n0, N, t * BK, ldw); };
    auto load_a = [&](int t) { load(stage(t), A, BM, m0, M, t * BK, lda); };
    // the weights of the first stages do not depend on the kernels ahead
    for (int t = 0; t < STAGES - 1; ++t)
        if (t < n_kt) load_w(t);
    pdl_wait();
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < n_kt) load_a(t);
        cp_async_commit();
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int tx = lane % 8 + 8 * (warp % (S::TX / 8)), ty = lane / 8 + 4 * (warp / (S::TX / 8));
    float acc[TM][TN];
#pragma unroll
    for (int i = 0; i < TM; ++i)
#pragma unroll
        for (int j = 0; j < TN; ++j) acc[i][j] = 0.f;
    for (int t = 0; t < n_kt; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        if (t + STAGES - 1 < n_kt) {
            load_w(t + STAGES - 1);
            load_a(t + STAGES - 1);
        }
        cp_async_commit();
        const float *as = stage(t) + ty * LD, *ws = stage(t) + (BM + tx) * LD;
#pragma unroll
        for (int k = 0; k < BK; k += 4) {
            float4 w[TN];
#pragma unroll
            for (int j = 0; j < TN; ++j) w[j] = *reinterpret_cast<const float4 *>(ws + j * S::TX * LD + k);
#pragma unroll
            for (int i = 0; i < TM; ++i) {
                const float4 a = *reinterpret_cast<const float4 *>(as + i * S::TY * LD + k);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.x, w[j].x, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.y, w[j].y, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.z, w[j].z, acc[i][j]);
#pragma unroll
                for (int j = 0; j < TN; ++j) acc[i][j] = fmaf(a.w, w[j].w, acc[i][j]);
            }
        }
    }
    pdl_trigger();      // at the end: the blocks of a product fill their SMs
#pragma unroll
    for (int j = 0; j < TN; ++j) {
        const int n = n0 + tx + j * S::TX;
        if (n >= N) continue;
        const float b = bias ? bias[n] : 0.f;
#pragma unroll
        for (int i = 0; i < TM; ++i) {
            const int m = m0 + ty + i * S::TY;
            if (m < M) C[(size_t)m * ldc + n] = from_f32<TO>(bias ? acc[i][j] + b : acc[i][j]);
        }
    }
}

// ---- tiles of rows that do not all start on 16 bytes ---------------------------------------------
constexpr int RAGGED_BM = 64, RAGGED_BN = 64, RAGGED_BK = 16, RAGGED_TM = 4, RAGGED_TN = 4;

template <typename TO>
__global__ void __launch_bounds__(256) gemm_f32_ragged_kernel(const float *__restrict__ A, const float *__restrict__ W,
                                                       const float *__restrict__ bias, TO *__restrict__ C, int M, int N, int K,
                                                       int lda, int ldw, int ldc) {
    pdl_trigger();
    pdl_wait();
    __shared__ float As[RAGGED_BK][RAGGED_BM + 4];
    __shared__ float Ws[RAGGED_BK][RAGGED_BN + 4];
    const int tid = threadIdx.x;
    const int tx = tid % 16, ty = tid / 16;  // thread's 4x4 patch: rows ty*4.., cols tx*4..
    const int m0 = blockIdx.y * RAGGED_BM, n0 = blockIdx.x * RAGGED_BN;
    float acc[RAGGED_TM][RAGGED_TN];
#pragma unroll
    for (int i = 0; i < RAGGED_TM; ++i)
#pragma unroll
        for (int j = 0; j < RAGGED_TN; ++j) acc[i][j] = 0.f;

    // each thread loads 4 elements of each tile: row = tid / 4 (0..63), k = (tid % 4) * 4 .. +3
    const int lr = tid / 4, lk = (tid % 4) * 4;
    for (int k0 = 0; k0 < K; k0 += RAGGED_BK) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const int k = k0 + lk + j;
            const int am = m0 + lr, wn = n0 + lr;
            As[lk + j][lr] = (am < M && k < K) ? act_load(A + (size_t)am * lda + k) : 0.f;
            Ws[lk + j][lr] = (wn < N && k < K) ? W[(size_t)wn * ldw + k] : 0.f;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < RAGGED_BK; ++k) {
            float a[RAGGED_TM], w[RAGGED_TN];
#pragma unroll
            for (int i = 0; i < RAGGED_TM; ++i) a[i] = As[k][ty * RAGGED_TM + i];
#pragma unroll
            for (int j = 0; j < RAGGED_TN; ++j) w[j] = Ws[k][tx * RAGGED_TN + j];
#pragma unroll
            for (int i = 0; i < RAGGED_TM; ++i)
#pragma unroll
                for (int j = 0; j < RAGGED_TN; ++j) acc[i][j] = fmaf(a[i], w[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < RAGGED_TM; ++i) {
        const int m = m0 + ty * RAGGED_TM + i;
        if (m >= M) continue;
#pragma unroll
        for (int j = 0; j < RAGGED_TN; ++j) {
            const int n = n0 + tx * RAGGED_TN + j;
            if (n >= N) continue;
            float v = acc[i][j];
            if (bias) v += bias[n];
            C[(size_t)m * ldc + n] = from_f32<TO>(v);
        }
    }
}

// ---- products of a long K: eight tensor-core products of three parts each -------------------------
// A run of 16 k is added up by add_run (bf16_thirds.cuh; 16 features by 8 rows), the run's sums join the sum of its segment of 128 k in
// float32, and the segments' sums join in order.  One order for every kernel below, so a row has the same bits in each.  A result that is
// not finite, or below 2^-96, is formed again as the plain chain of FMAs: infinities, NaNs and overflows come out as they do there, and so
// do sums of numbers so small that a part is cut (a bfloat16 number below the normal ones is a multiple of 2^-133, so an operand
// under 2^-110 has fewer than 24 bits; that shows in larger results beside operands over 2^14 only).
constexpr int SEGMENT = 128, SPLIT_FROM = 64;

__device__ __forceinline__ bool by_chain(float v) { return !(fabsf(v) <= 3.402823466e38f) || (fabsf(v) < 0x1p-96f && v != 0.f); }

// The chains of a block that has such a result, of all its outputs side by side: FEATURES rows of W and ROWS of A come through shared memory STEP
// elements at a time, and add(w, a) has every thread's FMAs of one k (row r's at w[r (STEP + 1)]).  One thread's chain after another, from memory,
// took up to 40 times as long as a product without (812 x 11,264 x 2,048 with a NaN in every row: 26,000 us, 2,500 here, 860 without one; 4 rows 320,
// 155 and 40).
template <int FEATURES, int ROWS, int THREADS, int STEP, typename Add>
__device__ __forceinline__ void chain_tile(const float *A, const float *W, int m0, int n0, int M, int N, int K, int lda, int ldw, float *ws, Add &&add) {
    constexpr int LD = STEP + 1, EACH = (FEATURES + ROWS) * STEP / THREADS, NOW = EACH % 8 ? 6 : 8;
    static_assert((FEATURES + ROWS) * STEP % THREADS == 0 && EACH % NOW == 0, "whole rounds of loads");
    cp_async_wait<0>();
#pragma unroll 1
    for (int k0 = 0; k0 < K; k0 += STEP) {
        const int n = min(STEP, K - k0);
        __syncthreads();
#pragma unroll 1
        for (int i0 = 0; i0 < EACH; i0 += NOW) {
            float v[NOW];
#pragma unroll
            for (int i = 0; i < NOW; ++i) {
                const int at = (i0 + i) * THREADS + threadIdx.x, r = at / STEP, k = min(at % STEP, n - 1);
                v[i] = act_load(r < FEATURES ? W + (size_t)min(n0 + r, N - 1) * ldw + k0 + k : A + (size_t)min(m0 + r - FEATURES, M - 1) * lda + k0 + k);
            }
#pragma unroll
            for (int i = 0; i < NOW; ++i) {
                const int at = (i0 + i) * THREADS + threadIdx.x;
                ws[at / STEP * LD + at % STEP] = v[i];
            }
        }
        __syncthreads();
#pragma unroll 8
        for (int i = 0; i < n; ++i) add(ws + i, ws + FEATURES * LD + i);
    }
}

template <typename TO>
__device__ __forceinline__ void store_split(float v, const float *bias, TO *C, int m, int n, int M, int N, int ldc) {
    if (m < M && n < N) C[(size_t)m * ldc + n] = from_f32<TO>(bias ? v + bias[n] : v);
}

// 16 bytes of a row's elements k .. k + 3 into shared memory, zeros for those past K.  Rows that do not start on 16 bytes come
// element by element (through L1: such a kernel is launched without the early start).
template <bool VEC> __device__ __forceinline__ void copy_4(uint32_t dst, const float *src, int k, int K) {
    const int n = min(max(K - k, 0), 4);
    if constexpr (VEC) {
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(n ? src : src - k), "r"(n * 4) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(dst + 4 * i), "l"(i < n ? src + i : src - k), "r"(i < n ? 4 : 0) : "memory");
    }
}
// ROWS rows of 32 floats, k0 on, by THREADS threads of eight a row.  `x` is the first row at this thread's 16 bytes of it; off[] are its rows.
// The halves of every second row change places in shared memory, so that eight lanes' 16-byte reads of one half of two rows fall
// into all 32 banks.
template <bool VEC> using RowOffset = typename std::conditional<VEC, int, long long>::type;
template <bool VEC, int ROWS, int THREADS>
__device__ __forceinline__ void copy_rows(uint32_t dst, const float *x, const RowOffset<VEC> (&off)[ROWS * 8 / THREADS], int k0, int c, int K, int rows = ROWS) {
    constexpr int N = ROWS * 8 / THREADS, BYTES = THREADS / 8 * 128;
    if (VEC && k0 + 32 <= K) {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i * (THREADS / 8) < rows) asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + i * BYTES), "l"(x + k0 + off[i]) : "memory");
    } else {
#pragma unroll
        for (int i = 0; i < N; ++i)
            if (i * (THREADS / 8) < rows) copy_4<VEC>(dst + i * BYTES, x + k0 + off[i], k0 + c, K);
    }
}
__device__ __forceinline__ int swizzled(int row, int chunk) { return row * 32 + ((chunk ^ ((row & 1) << 2)) << 2); }

// Few rows: a block has 16 features and up to 8 NT rows; its eight warps take a segment of K each, turn by turn, and stream W
// through shared memory of their own (no barrier but at the end of a turn).  Rows that are not there repeat the last one.
constexpr int FEW_EACH = 4, SEGMENT_STEPS = SEGMENT / 32;
template <int NT, int STAGES, int WARPS> struct FewShape {
    static constexpr int STAGE_FLOATS = (16 + 8 * NT) * 32;
    static constexpr int OUTS = NT * 128;               // of a block
    static constexpr size_t SMEM = sizeof(float) * (WARPS * STAGES * STAGE_FLOATS + WARPS * FEW_EACH * OUTS);
};

template <int NT, int STAGES, int WARPS, bool VEC, typename TO>
__global__ void __launch_bounds__(WARPS * 32) gemm_f32_few_kernel(const float *__restrict__ A, const float *__restrict__ W,
                                                                      const float *__restrict__ bias, TO *__restrict__ C, int M, int N, int K, int lda,
                                                                      int ldw, int ldc) {
    using S = FewShape<NT, STAGES, WARPS>;
    constexpr int SEGS = WARPS * FEW_EACH;                                           // segments of the block in a turn
    static_assert(SEGMENT_STEPS % STAGES == 0, "a step's stage is known when it is compiled");
    extern __shared__ __align__(16) float smem_f[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int n0 = blockIdx.x * 16, m0 = blockIdx.y * 8 * NT;
    float *mine = smem_f + warp * STAGES * S::STAGE_FLOATS, *parts = smem_f + WARPS * STAGES * S::STAGE_FLOATS;
    const int n_seg = (K + SEGMENT - 1) / SEGMENT;
    const int r = lane >> 3, c = (lane & 7) * 4;
    const float *wp = W + (size_t)n0 * ldw + c, *ap = A + (size_t)m0 * lda + c;
    RowOffset<VEC> w_off[4], a_off[2 * NT];
#pragma unroll
    for (int i = 0; i < 4; ++i) w_off[i] = (RowOffset<VEC>)min(i * 4 + r, N - 1 - n0) * ldw;
#pragma unroll
    for (int i = 0; i < 2 * NT; ++i) a_off[i] = (RowOffset<VEC>)min(i * 4 + r, M - 1 - m0) * lda;
    const uint32_t to = smem_addr(mine + swizzled(r, lane & 7));
    // step s of a turn that starts at segment `first`: 32 k of this warp's segment s / SEGMENT_STEPS; behind its last the next turn's
    auto k_of = [&](int first, int s) { return (first + s / SEGMENT_STEPS * WARPS + warp) * SEGMENT + s % SEGMENT_STEPS * 32; };
    auto load_w = [&](int k0, int s) {
        if (k0 < K) copy_rows<VEC, 16, 32>(to + (s % STAGES) * S::STAGE_FLOATS * 4, wp, w_off, k0, c, K);
    };
    auto load_a = [&](int k0, int s) {
        if (k0 < K) copy_rows<VEC, 8 * NT, 32>(to + ((s % STAGES) * S::STAGE_FLOATS + 16 * 32) * 4, ap, a_off, k0, c, K, M - m0);
    };
    // the weights of the first stages do not depend on the kernels ahead
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) load_w(k_of(0, s), s);
    pdl_wait();
#pragma unroll
    for (int s = 0; s < STAGES - 1; ++s) {
        load_a(k_of(0, s), s);
        cp_async_commit();
    }
    constexpr int OUTS = (S::OUTS + WARPS * 32 - 1) / (WARPS * 32);         // ... of a thread
    float total[OUTS];
#pragma unroll
    for (int o = 0; o < OUTS; ++o) total[o] = 0.f;
    const int frag = swizzled(g, q), frag_other = frag ^ 16;          // the row's first and second 16 k (rows 8 apart have the same order)
    for (int first = 0; first < n_seg; first += SEGS) {
        // (loops, not 32 copies of a step: a step is up to 500 instructions, and blocks that start would wait for them from memory; 32 x 2,048 x 5,632:
        // 53 us with all 16 steps of a turn in a row)
#pragma unroll 1
        for (int i = 0; i < FEW_EACH; ++i) {
            if (first + i * WARPS + warp >= n_seg) break;
            float sum[1][NT][4];
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) sum[0][j][e] = 0.f;
#pragma unroll(NT <= 2 ? SEGMENT_STEPS / STAGES : 1)
            for (int s0 = i * SEGMENT_STEPS; s0 < (i + 1) * SEGMENT_STEPS; s0 += STAGES) {
#pragma unroll
                for (int u = 0; u < STAGES; ++u) {          // (the step's stage)
                    const int s = s0 + u, k0 = k_of(first, s), ahead = s + STAGES - 1;
                    cp_async_wait<STAGES - 2>();
                    __syncwarp();
                    load_w(k_of(first, ahead), u + STAGES - 1);
                    load_a(k_of(first, ahead), u + STAGES - 1);
                    cp_async_commit();
                    const float *ws = mine + u * S::STAGE_FLOATS;
                    if (k0 < K) {
#pragma unroll
                        for (int run = 0; run < 2; ++run) {
                            const float *at = ws + (run ? frag_other : frag);
                            float4 w[1][2], a[NT];
                            w[0][0] = *reinterpret_cast<const float4 *>(at);
                            w[0][1] = *reinterpret_cast<const float4 *>(at + 8 * 32);
#pragma unroll
                            for (int j = 0; j < NT; ++j) a[j] = *reinterpret_cast<const float4 *>(at + (16 + j * 8) * 32);
                            add_run<1, NT>(sum, w, a);
                        }
                    }
                    __syncwarp();
                }
            }
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) parts[(i * WARPS + warp) * S::OUTS + (j * 4 + e) * 32 + lane] = sum[0][j][e];
        }
        // the turn's segments, in order
        __syncthreads();
        const int segs = min(SEGS, n_seg - first);
#pragma unroll
        for (int o = 0; o < OUTS; ++o) {
            const int at = o * WARPS * 32 + threadIdx.x;
            if (at < S::OUTS) {
#pragma unroll 8
                for (int s = 0; s < segs; ++s) total[o] += parts[s * S::OUTS + at];
            }
        }
        if (first + SEGS < n_seg) __syncthreads();
    }
    pdl_trigger();      // at the end: blocks of the kernels behind that start earlier are placed where there is room, not where there is time
    // an output of a thread: its feature and its row in the block
    auto feature = [&](int o) { return ((o * WARPS * 32 + (int)threadIdx.x) & 31) / 4 + (((o * WARPS * 32 + (int)threadIdx.x) >> 6) & 1) * 8; };
    auto row = [&](int o) { return (o * WARPS * 32 + (int)threadIdx.x) / 128 * 8 + (threadIdx.x & 3) * 2 + (((o * WARPS * 32 + (int)threadIdx.x) >> 5) & 1); };
    auto there = [&](int o) { return o * WARPS * 32 + (int)threadIdx.x < S::OUTS && m0 + row(o) < M && n0 + feature(o) < N; };
    bool again = false;
#pragma unroll
    for (int o = 0; o < OUTS; ++o) again |= there(o) && by_chain(total[o]);
    if (__syncthreads_or(again)) {
        float v[OUTS] = {};
        constexpr int STEP = 128, LD = STEP + 1;
        chain_tile<16, 8 * NT, WARPS * 32, STEP>(A, W, m0, n0, M, N, K, lda, ldw, smem_f, [&](const float *w, const float *a) {
#pragma unroll
            for (int o = 0; o < OUTS; ++o)
                if (there(o)) v[o] = fmaf(a[row(o) * LD], w[feature(o) * LD], v[o]);
        });
#pragma unroll
        for (int o = 0; o < OUTS; ++o)
            if (by_chain(total[o])) total[o] = v[o];
    }
#pragma unroll
    for (int o = 0; o < OUTS; ++o)
        if (there(o)) store_split(total[o], bias, C, m0 + row(o), n0 + feature(o), M, N, ldc);
}

// Many rows: tiles of 64 features by 64 rows, 32 x 32 a warp.  The tensor pipe and the schedulers bound it: a product of m16n8k16 holds its
// scheduler for nearly nine cycles (560 TFLOP/s by itself, eight a product: 596 of the 861 us of 812 x 11,264 x 2,048), the parts and sums take
// the rest.  A segment's sum and the sum of segments stay in registers.
constexpr int MANY_STAGES = 4, MANY_STAGE_FLOATS = 128 * 32;
constexpr size_t MANY_SMEM = sizeof(float) * MANY_STAGES * MANY_STAGE_FLOATS;

template <bool VEC, typename TO>
__global__ void __launch_bounds__(128, 3) gemm_f32_many_kernel(const float *__restrict__ A, const float *__restrict__ W, const float *__restrict__ bias,
                                                               TO *__restrict__ C, int M, int N, int K, int lda, int ldw, int ldc, int tiles_m) {
    constexpr int STAGES = MANY_STAGES;
    extern __shared__ __align__(16) float smem_f[];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    const int f0 = (warp & 1) * 32, r0 = (warp >> 1) * 32;
    // row tiles fastest: the blocks that run at one time share a few tiles of W, and A stays in L2
    const int m0 = (int)(blockIdx.x % tiles_m) * 64, n0 = (int)(blockIdx.x / tiles_m) * 64;
    const int n_kt = (K + 31) / 32;
    const int r = threadIdx.x >> 3, c = (threadIdx.x & 7) * 4;
    const float *wp = W + (size_t)n0 * ldw + c, *ap = A + (size_t)m0 * lda + c;
    RowOffset<VEC> w_off[4], a_off[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        w_off[i] = (RowOffset<VEC>)min(i * 16 + r, N - 1 - n0) * ldw;
        a_off[i] = (RowOffset<VEC>)min(i * 16 + r, M - 1 - m0) * lda;
    }
    const uint32_t to = smem_addr(smem_f + swizzled(r, threadIdx.x & 7));
    auto load_w = [&](int t) { copy_rows<VEC, 64, 128>(to + (t % STAGES) * MANY_STAGE_FLOATS * 4, wp, w_off, t * 32, c, K); };
    auto load_a = [&](int t) { copy_rows<VEC, 64, 128>(to + ((t % STAGES) * MANY_STAGE_FLOATS + 64 * 32) * 4, ap, a_off, t * 32, c, K); };
    // the weights of the first stages do not depend on the kernels ahead
    for (int t = 0; t < STAGES - 1; ++t)
        if (t < n_kt) load_w(t);
    pdl_wait();
    for (int t = 0; t < STAGES - 1; ++t) {
        if (t < n_kt) load_a(t);
        cp_async_commit();
    }
    float sum[2][4][4], total[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[i][j][e] = total[i][j][e] = 0.f;
    const int frag = swizzled(g, q);
    for (int t = 0; t < n_kt; ++t) {
        cp_async_wait<STAGES - 2>();
        __syncthreads();
        if (t + STAGES - 1 < n_kt) {
            load_w(t + STAGES - 1);
            load_a(t + STAGES - 1);
        }
        cp_async_commit();
        const float *st = smem_f + (t % STAGES) * MANY_STAGE_FLOATS;
#pragma unroll
        for (int run = 0; run < 2; ++run) {
            if (run == 0 || t * 32 + 16 < K) {
                const float *ws = st + f0 * 32 + (frag ^ (run * 16)), *as = st + (64 + r0) * 32 + (frag ^ (run * 16));
                float4 w[2][2], a[4];
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int h = 0; h < 2; ++h) w[i][h] = *reinterpret_cast<const float4 *>(ws + (i * 16 + h * 8) * 32);
#pragma unroll
                for (int j = 0; j < 4; ++j) a[j] = *reinterpret_cast<const float4 *>(as + j * 8 * 32);
                add_run<2, 4>(sum, w, a);
            }
        }
        if (t % (SEGMENT / 32) == SEGMENT / 32 - 1 || t + 1 == n_kt) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e) {
                        total[i][j][e] += sum[i][j][e];
                        sum[i][j][e] = 0.f;
                    }
        }
    }
    pdl_trigger();      // at the end: the blocks of a product fill their SMs
    const int row = r0 + q * 2, feature = f0 + g;               // of output (i, j, e): row + 8 j + e % 2, feature + 16 i + 8 (e / 2)
    bool again = false;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) again |= m0 + row + 8 * j + (e & 1) < M && n0 + feature + 16 * i + 8 * (e >> 1) < N && by_chain(total[i][j][e]);
    if (__syncthreads_or(again)) {
        float v[2][4][4] = {};
        constexpr int STEP = 64, LD = STEP + 1;
        chain_tile<64, 64, 128, STEP>(A, W, m0, n0, M, N, K, lda, ldw, smem_f, [&](const float *w, const float *a) {
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        v[i][j][e] = fmaf(a[(row + 8 * j + (e & 1)) * LD], w[(feature + 16 * i + 8 * (e >> 1)) * LD], v[i][j][e]);
        });
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e)
                    if (by_chain(total[i][j][e])) total[i][j][e] = v[i][j][e];
    }
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) store_split(total[i][j][e], bias, C, m0 + row + 8 * j + (e & 1), n0 + feature + 16 * i + 8 * (e >> 1), M, N, ldc);
}

// ---- host side -----------------------------------------------------------------------------------
// (At every launch: the attribute belongs to the kernel on the current device, and a process may use several.)
template <typename Kernel> int allow_smem(Kernel kernel, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) LGML_FAIL("gemm_f32: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    return 0;
}

struct Call {
    const float *A, *W, *bias;
    void *C;
    int M, N, K, lda, ldw, ldc;
    cudaStream_t stream;
};

// Products of this many multiply-adds a row and more are launched alone: their blocks are few an SM and as long as K, so where
// they lie decides (four requests at width 2,048: 24 us a product of N or K 2,048 with the attribute, 19 without).  Smaller ones
// end within a few microseconds, of which an early start is a part.
bool balanced(const Call &c) { return (long long)c.N * c.K >= 1 << 21; }

template <int F, int MT, bool VEC, typename TO> int launch_rows(const Call &c) {
    auto kernel = gemm_f32_rows_kernel<F, MT, VEC, TO>;
    if (allow_smem(kernel, RowsShape<F, MT>::SMEM)) return -1;
    const dim3 grid((unsigned)((c.N + F - 1) / F));
    if (balanced(c)) lgml_launch_alone(kernel, grid, 32, RowsShape<F, MT>::SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    else lgml_launch(kernel, grid, 32, RowsShape<F, MT>::SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    return lgml_launch_status("gemm_f32");
}

template <int BM, int BN, int TM, int TN, typename TO> int launch_tiles(const Call &c) {
    using S = TileShape<BM, BN, TM, TN>;
    auto kernel = gemm_f32_tile_kernel<BM, BN, TM, TN, TO>;
    if (allow_smem(kernel, S::SMEM)) return -1;
    const int tiles_m = (c.M + BM - 1) / BM;
    const long long tiles = (long long)tiles_m * ((c.N + BN - 1) / BN);
    if (tiles > 0x7fffffffLL) LGML_FAIL("gemm_f32: M=%d N=%d make too many tiles", c.M, c.N);
    const dim3 grid((unsigned)tiles);
    if (balanced(c)) lgml_launch_alone(kernel, grid, S::THREADS, S::SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, tiles_m);
    else lgml_launch(kernel, grid, S::THREADS, S::SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, tiles_m);
    return lgml_launch_status("gemm_f32");
}
template <typename TO> int launch_ragged(const Call &c) {
    const dim3 grid((c.N + RAGGED_BN - 1) / RAGGED_BN, (c.M + RAGGED_BM - 1) / RAGGED_BM);
    lgml_launch(gemm_f32_ragged_kernel<TO>, grid, 256, 0, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    return lgml_launch_status("gemm_f32");
}

// Features a warp for M <= 4 rows: eight where that is one warp for each of the chip's 592 schedulers or fewer.
template <bool VEC, typename TO> int run_rows(const Call &c) {
    if (c.N <= 592 * 8) return launch_rows<8, 1, VEC, TO>(c);
    return c.M <= 2 ? launch_rows<16, 1, VEC, TO>(c) : launch_rows<16, 2, VEC, TO>(c);
}

// Time of a product on tiles of bm x bn, in microseconds at K = 2048, where the shapes were first compared: an SM's first tile takes `alone`
// (one block does not fill the FMA units), every further one `more`.  For 5 to 2,000 rows of 512 to 32,000 features and K of 4 to 60 the shape that it says is
// within 5 % of the best of the four on average, 27 % at worst; one shape for all sizes is 8 % (32 x 64) to 47 % (64 x 128) behind on average.
float tiled_us(const Call &c, int bm, int bn, float alone, float more) {
    const long long tiles = (long long)((c.M + bm - 1) / bm) * ((c.N + bn - 1) / bn);
    return alone + (float)((tiles + 147) / 148 - 1) * more;
}

template <int NT, int STAGES, int WARPS, bool VEC, typename TO> int launch_few(const Call &c) {
    auto kernel = gemm_f32_few_kernel<NT, STAGES, WARPS, VEC, TO>;
    constexpr size_t smem = FewShape<NT, STAGES, WARPS>::SMEM;
    if (allow_smem(kernel, smem)) return -1;
    const dim3 grid((unsigned)((c.N + 15) / 16), (unsigned)((c.M + 8 * NT - 1) / (8 * NT)));
    // decoding's products start early: their first weights come while the kernel ahead ends (about 2 us each)
    if (!VEC || NT > 2) lgml_launch_alone(kernel, grid, WARPS * 32, smem, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    else lgml_launch(kernel, grid, WARPS * 32, smem, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc);
    return lgml_launch_status("gemm_f32");
}
template <bool VEC, typename TO> int launch_many(const Call &c) {
    auto kernel = gemm_f32_many_kernel<VEC, TO>;
    if (allow_smem(kernel, MANY_SMEM)) return -1;
    const int tiles_m = (c.M + 63) / 64;
    const long long tiles = (long long)tiles_m * ((c.N + 63) / 64);
    if (tiles > 0x7fffffffLL) LGML_FAIL("gemm_f32: M=%d N=%d make too many tiles", c.M, c.N);
    const dim3 grid((unsigned)tiles);
    if (!VEC || balanced(c)) lgml_launch_alone(kernel, grid, 128, MANY_SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, tiles_m);
    else lgml_launch(kernel, grid, 128, MANY_SMEM, c.stream, c.A, c.W, c.bias, (TO *)c.C, c.M, c.N, c.K, c.lda, c.ldw, c.ldc, tiles_m);
    return lgml_launch_status("gemm_f32");
}
// Time of a product on blocks of 16 features by 32 rows, and on tiles of 64 by 64, in microseconds at K = 2048: a round of blocks
// takes 12.5; an SM's first tile takes 70 (one warp a scheduler), every further one 53.
template <bool VEC, typename TO> int run_split(const Call &c) {
    // Where there is one block an SM it has sixteen warps, else two blocks share the SM (4 rows, N x K, sixteen warps and eight:
    // 2048 x 5632 12.3 and 15.5, 2048 x 2048 6.3 and 6.9, 3072 x 2048 11.2 and 9.3, 11264 x 2048 28.5 and 22.3; 16 rows 16.6 and 21.9, 7.3 and 8.7, 13.8
    // and 12.7, 34.2 and 30.3).
    const bool one = c.N <= 148 * 16;
    if (c.M <= 8) return one ? launch_few<1, 4, 16, VEC, TO>(c) : launch_few<1, 4, 8, VEC, TO>(c);
    if (c.M <= 16) return one ? launch_few<2, 2, 16, VEC, TO>(c) : launch_few<2, 2, 8, VEC, TO>(c);
    const long long blocks = (long long)((c.M + 31) / 32) * ((c.N + 15) / 16), tiles = (long long)((c.M + 63) / 64) * ((c.N + 63) / 64);
    // (the blocks' rows are the grid's second dimension: no more than 65,535 of them)
    if ((blocks + 147) / 148 * 12.5f <= 70 + ((tiles + 147) / 148 - 1) * 53 && c.M <= 65535 * 32) return launch_few<4, 2, 8, VEC, TO>(c);
    return launch_many<VEC, TO>(c);
}

// A short K as chains of FMAs.  Tiles, but for one and two rows of K > 32, or four of up to 1,024 features (four rows of 512, K 60: 1.5 us, in tiles
// 2.1; two rows here and there: K 60, 512 features 1.3 and 2.1 us, 8,192 2.1 and 3.0,
// 32,000 5.0 and 6.5; K 32, 2,048 features 1.8 and 1.6, 32,000 4.7 and 3.9; four rows, K 48: 2.2 and 1.9, 32,000 6.2 and 5.1).  Element by element the
// tiles are slower (8 rows of 8,192 features, K 48: 6.8 us, in tiles of 16-byte copies 2.6), so rows that do not start on 16 bytes keep warps of their own up
// to four, but not of a vocabulary's size (4 rows of N 30000, K 31: 8.8 and 7.3).
template <bool VEC, typename TO> int run(const Call &c) {
    if (c.K >= SPLIT_FROM) return run_split<VEC, TO>(c);
    if (VEC ? c.K > 32 && c.M <= (c.N <= 1024 ? 4 : 2) : c.M <= 4 && c.N <= 148 * 128) return run_rows<VEC, TO>(c);
    if constexpr (VEC) {
        const float t1 = tiled_us(c, 32, 32, 40.f, 19.6f), t2 = tiled_us(c, 32, 64, 58.f, 32.f), t3 = tiled_us(c, 64, 64, 90.f, 58.7f),
                    t4 = tiled_us(c, 64, 128, 148.f, 108.f);
        if (t4 <= t1 && t4 <= t2 && t4 <= t3) return launch_tiles<64, 128, 8, 8, TO>(c);
        if (t3 <= t1 && t3 <= t2) return launch_tiles<64, 64, 8, 4, TO>(c);
        return t2 <= t1 ? launch_tiles<32, 64, 4, 4, TO>(c) : launch_tiles<32, 32, 4, 2, TO>(c);
    } else {
        return launch_ragged<TO>(c);
    }
}
}  // namespace

// out_dtype selects the type C is stored in; the sum itself is float32 in both cases.
LGML_API int lgml_gemm_f32(const float *A, const float *W, const float *bias, void *C, int out_dtype, int M, int N, int K,
                           int lda, int ldw, int ldc, cudaStream_t stream) {
    LGML_REQUIRE(M >= 0 && N > 0 && K > 0, "gemm_f32: bad sizes M=%d N=%d K=%d", M, N, K);
    LGML_REQUIRE(lda >= K && ldw >= K && ldc >= N, "gemm_f32: a leading dimension is smaller than its row");
    if (M == 0) return 0;
    LGML_REQUIRE((M + 63) / 64 <= 65535, "gemm_f32: M=%d is over %d rows", M, 65535 * 64);
    const Call c = {A, W, bias, C, M, N, K, lda, ldw, ldc, stream};
    // 16-byte copies need rows that start on 16 bytes, and a tile's rows within 31 bits; any other matrix goes element by element
    const bool vec = lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0 && lda <= 1 << 25 && ldw <= 1 << 25;
    if (out_dtype == LGML_F32) return vec ? run<true, float>(c) : run<false, float>(c);
    if (out_dtype == LGML_BF16) return vec ? run<true, __nv_bfloat16>(c) : run<false, __nv_bfloat16>(c);
    LGML_FAIL("gemm_f32: unknown output type %d", out_dtype);
}
