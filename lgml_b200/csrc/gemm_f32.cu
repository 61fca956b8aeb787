// True 32-bit matrix product: C[M,N] = A[M,K] . W[N,K]^T (+ bias[N]), float32 operands,
// float32 FMA accumulation, no tensor cores and no reduced-precision mode.  Every output
// element sums its K products in the order k = 0, 1, 2, ... whatever M, N and the tile it
// falls in, so a row's result does not depend on what else is in the batch.  It stands
// where mischief/lgml calls mul_mat with the f32 flag (src/lgml.c:1811-1839).
//
// That order makes one chain of K dependent FMAs of every output (4 cycles each: 8.5 us at
// K = 4096), so K is never cut; the kernels differ in what they keep busy beside the chain:
//   * gemm_f32_rows_kernel, up to 16 rows (decoding): the matrix is what has to be read.  A warp
//     streams 8 to 32 rows of W through shared memory of its own, a lane owns one feature for a few
//     rows; the first stages are asked for before the kernel ahead is done.
//   * gemm_f32_tile_kernel, more rows: tiles of A and W by asynchronous copies, several blocks an SM.
//   * gemm_f32_ragged_kernel, more rows that do not all start on 16 bytes: tiles element by element.
// One B200, weights from HBM, microseconds before (64 x 64 tiles, element by element) and now:
//   M, N, K:  4, 2048, 2048: 156 -> 13;  4, 11264, 2048: 225 -> 26;  4, 32000, 2048: 435 -> 59;
//   89, 2048, 5632: 423 -> 158;  512, 11264, 2048: 998 -> 554 (43 TFLOP/s);  1500, 32000, 2048: 7927 -> 4388.
// From registers alone (16 independent chains a thread) the FMA units give 72 TFLOP/s.

#include "common.cuh"

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
        if constexpr (MT <= 4) {
            constexpr int AHEAD = MT <= 2 ? 4 : 2, GROUPS = ROWS_BK / 4 / AHEAD;
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
        } else {
#pragma unroll 8
            for (int k = 0; k < ROWS_BK; k += 4) {
                float4 w, a[MT];
                read(k, w, a);
                add(w, a);
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

// Features a warp for M <= 16 rows.  Eight where that is one warp for each of the chip's 592 schedulers or
// fewer (N 2048, K 2048: 12.5 us at 4 rows; 15 with sixteen, 21 with thirty-two); more features beside a
// reading of A as soon as there are warps enough (N 11264, 4 rows: 38, 26 and 29 us; 8 rows: 45, 49 and 36).
template <bool VEC, typename TO> int run_rows(const Call &c) {
    if (c.N <= 592 * 8) return c.M <= 4 ? launch_rows<8, 1, VEC, TO>(c) : (c.M <= 8 ? launch_rows<8, 2, VEC, TO>(c) : launch_rows<8, 4, VEC, TO>(c));
    if (c.M <= 4) return c.M <= 2 ? launch_rows<16, 1, VEC, TO>(c) : launch_rows<16, 2, VEC, TO>(c);
    return c.M <= 8 ? launch_rows<32, 8, VEC, TO>(c) : launch_rows<32, 16, VEC, TO>(c);
}

// Time of a product on tiles of bm x bn, in microseconds at K = 2048: an SM's first tile takes `alone`
// (one block does not fill the FMA units), every further one `more`.
float tiled_us(const Call &c, int bm, int bn, float alone, float more) {
    const long long tiles = (long long)((c.M + bm - 1) / bm) * ((c.N + bn - 1) / bn);
    return alone + (float)((tiles + 147) / 148 - 1) * more;
}

// Whether up to 16 rows go to warps of their own.  Not 9 to 16 rows of a vocabulary's size: a warp's reading of its rows of A, 145 to
// 170 us at N 32000, K 2048, costs more than what 32 x 32 tiles compute for rows that are not there, 149.  Not five rows and more of
// a short K, most of a stage being empty (N 4700, K 32: 3.3 to 4.5 us, 64 x 64 tiles element by element 3.0 to 3.3; K 64: 4.4 to 5.0, 5.2).
// Rows that do not start on 16 bytes come element by element here too, which a longer K, or fewer rows, must pay for
// (rows here, tiles; N 4700: 8 rows, K 31 4.1, 2.9, K 129 7.3, 9.0; 16 rows, K 129 10.2, 9.1, K 257 14.2, 16.3; N 18000: 8 rows,
// K 257 56.5, 51.9, K 513 79, 101; N 30000: 8 rows, K 257 83, 55, 4 rows, K 31 8.8, 7.3, K 129 27.1, 29.3).
template <bool VEC> bool rows_pay(const Call &c) {
    if (c.M > 16 || (c.M > 8 && c.N > 148 * 128)) return false;
    if (VEC) return c.M <= 4 || c.K >= 64;
    if (c.N > 148 * 128) return c.M <= 4 && c.K >= 64;
    return c.M <= 4 || c.K >= (c.N > 148 * 64 ? 512 : c.M <= 8 ? 64 : 256);
}

template <bool VEC, typename TO> int run(const Call &c) {
    if (rows_pay<VEC>(c)) return run_rows<VEC, TO>(c);
    if (VEC && c.M <= 16 && c.N <= 148 * 128) return launch_ragged<TO>(c);
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
    // 16-byte copies need rows that start on 16 bytes; any other matrix goes element by element
    const bool vec = lda % 4 == 0 && ldw % 4 == 0 && (((uintptr_t)A | (uintptr_t)W) & 15) == 0;
    if (out_dtype == LGML_F32) return vec ? run<true, float>(c) : run<false, float>(c);
    if (out_dtype == LGML_BF16) return vec ? run<true, __nv_bfloat16>(c) : run<false, __nv_bfloat16>(c);
    LGML_FAIL("gemm_f32: unknown output type %d", out_dtype);
}
