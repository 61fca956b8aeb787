// A selective state-space recurrence with a scalar decay per head ("state-space duality"):
//
//   dt_t = softplus(dt_raw_t + dt_bias_h)                       per head h
//   S_t  = exp(-exp(A_log_h) dt_t) S_(t-1) + dt_t B_t x_t^T      S is [N, P] per head; B, C are shared by the heads of a group
//   y_t  = S_t^T C_t + D_h x_t
//
//   ssd_scan       the recurrence over a step's tokens, request by request, S in the request's state slot; the same kernel
//                  runs S_t = a_t S_(t-1) + b_t B_t x_t^T with decays a and write weights b given per (token, head), with
//                  one column more than x has whose x is 1 (the sum of the written B, a normaliser) if asked for
//   ssd_gate_norm  (y silu(z)) over the root mean square of each of `groups` equal parts, times a weight
//
// Everything is float32 arithmetic in both compute types.  The state of a head is stored column by
// column ([P][N]): a thread owns a slice of one column and keeps it in registers over the step's tokens.
#include <math.h>

#include "common.cuh"
#include "bf16_thirds.cuh"

LGML_DEFINE_LAST_ERROR(lgml_ssd)

namespace {

constexpr int SCAN_THREADS = 128;

__device__ __forceinline__ float softplus_(float v) { return v > 20.f ? v : log1pf(expf(v)); }
__device__ __forceinline__ float silu_(float v) { return v / (1.0f + expf(-v)); }

// xbc float32 [n, ldx]: x of head h at column h P, B of group g at column x_cols + g N, C at x_cols + (G + g) N.
// dt_raw float32 [n, ldd], column h.  state: per slot [Hs][P][N].  y float32 [n, ldy], column h P + p.
// Block: (column tile, head, request).  A thread owns RN entries of each of CQ neighbouring columns: what it reads of
// a token's B and C serves CQ columns (the shared-memory reads are what bounds this kernel).  A column's N entries are
// dealt over LN neighbouring lanes in groups of four: lane l owns the groups l, l + LN, l + 2 LN ..., so the lanes
// read neighbouring 16-byte pieces of B and C from shared memory (no bank is asked twice) and of the state from memory.
// The step's tokens come through shared memory in groups of TT: B, C (rows of NS = LN RN floats, zeros behind N),
// the tile's x, dt and the decay.
// GIVEN: dt_raw holds the write weights themselves and a_given the decays (row stride ldd too); no skip term.  x has Px
// columns per head; columns Px .. P - 1 of the state are written with x = 1.  QUADS: the state's groups of four lie on 16 bytes.
template <int RN, int CQ, bool GIVEN, bool QUADS>
__global__ void __launch_bounds__(SCAN_THREADS) ssd_scan_kernel(const float *__restrict__ xbc, int ldx, const float *__restrict__ dt_raw, int ldd,
                                                                const float *__restrict__ dt_bias, const float *__restrict__ a_log,
                                                                const float *__restrict__ d_skip, float *__restrict__ state, long long state_ld,
                                                                const int *__restrict__ seq_start, const int *__restrict__ slots,
                                                                float *__restrict__ y, int ldy, int Hs, int G, int P, int N, int LN, int TT,
                                                                int pieces, int zero_start, float *__restrict__ decay_out, int vec,
                                                                const float *__restrict__ a_given, int Px, int max_tokens) {
    pdl_trigger();
    pdl_wait();
    if (max_tokens > 0 && seq_start[blockIdx.z + 1] - seq_start[blockIdx.z] > max_tokens) return;
    extern __shared__ float sm[];
    const int CPB = (SCAN_THREADS / LN) * CQ;          // columns of a block
    const int NS = LN * RN;
    float *Bs = sm, *Cs = Bs + (size_t)TT * NS, *xs = Cs + (size_t)TT * NS, *dts = xs + (size_t)TT * CPB, *dAs = dts + TT;
    const int h = blockIdx.y, s = blockIdx.z, g = h / (Hs / G);
    const int tid = threadIdx.x, col = tid / LN, ln = tid - col * LN;
    const int p0 = blockIdx.x * CPB + col * CQ;        // this thread's first column
    auto n_of = [&](int i) { return ((i >> 2) * LN + ln) * 4 + (i & 3); };      // the state entry behind this lane's i-th register
    // pieces: the step's tokens in pieces of consecutive tokens, rows (first, past the last) of an [n, 2] table
    const int t0 = pieces ? seq_start[2 * s] : seq_start[s], t1 = pieces ? seq_start[2 * s + 1] : seq_start[s + 1];
    const int x_cols = Hs * Px;
    const float a = GIVEN ? 0.f : expf(__ldg(a_log + h)), bias = GIVEN ? 0.f : __ldg(dt_bias + h), dsk = GIVEN ? 0.f : __ldg(d_skip + h);
    float *st = state + (size_t)(slots ? slots[s] : s) * state_ld + (size_t)h * P * N;
    float S[CQ][RN];
#pragma unroll
    for (int q = 0; q < CQ; ++q)
#pragma unroll
        for (int i = 0; i < RN; i += 4) {
            const float *at = st + (size_t)(p0 + q) * N + n_of(i);
            if (QUADS) {            // N a multiple of 4: a group is there or not as a whole
                const float4 v = (!zero_start && p0 + q < P && n_of(i) < N) ? act_load(reinterpret_cast<const float4 *>(at)) : make_float4(0.f, 0.f, 0.f, 0.f);
                S[q][i] = v.x, S[q][i + 1] = v.y, S[q][i + 2] = v.z, S[q][i + 3] = v.w;
            } else {
#pragma unroll
                for (int e = 0; e < 4; ++e) S[q][i + e] = (!zero_start && p0 + q < P && n_of(i) + e < N) ? act_load(at + e) : 0.f;
            }
        }
    float decay = 1.f;
    const bool want_y = y != nullptr;
    for (int tb = t0; tb < t1; tb += TT) {
        const int nt = min(TT, t1 - tb);
        __syncthreads();
        if (vec) {
            // 16 bytes a load, the loads of four rounds in flight before the first is stored
            const int NS4 = NS >> 2, N4 = N >> 2, total = nt * NS4;
            for (int i0 = tid; i0 < total; i0 += 4 * SCAN_THREADS) {
                float4 vb[4], vc[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + u * SCAN_THREADS;
                    vb[u] = vc[u] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (i < total) {
                        const int k = i / NS4, c = i - k * NS4;
                        if (c < N4) {
                            const float *rowp = xbc + (size_t)(tb + k) * ldx + x_cols;
                            vb[u] = act_load(reinterpret_cast<const float4 *>(rowp + (size_t)g * N) + c);
                            vc[u] = act_load(reinterpret_cast<const float4 *>(rowp + (size_t)(G + g) * N) + c);
                        }
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const int i = i0 + u * SCAN_THREADS;
                    if (i < total) reinterpret_cast<float4 *>(Bs)[i] = vb[u], reinterpret_cast<float4 *>(Cs)[i] = vc[u];
                }
            }
        } else {
            for (int i = tid; i < nt * NS; i += SCAN_THREADS) {
                const int k = i / NS, c = i - k * NS;
                const float *rowp = xbc + (size_t)(tb + k) * ldx + x_cols;
                Bs[i] = c < N ? act_load(rowp + (size_t)g * N + c) : 0.f;
                Cs[i] = c < N ? act_load(rowp + (size_t)(G + g) * N + c) : 0.f;
            }
        }
        for (int i = tid; i < nt * CPB; i += SCAN_THREADS) {
            const int k = i / CPB, c = i - k * CPB;
            const int pc = blockIdx.x * CPB + c;
            xs[k * CPB + c] = pc < Px ? act_load(xbc + (size_t)(tb + k) * ldx + (size_t)h * Px + pc) : (GIVEN && pc < P ? 1.f : 0.f);
        }
        for (int k = tid; k < nt; k += SCAN_THREADS) {
            const float raw = act_load(dt_raw + (size_t)(tb + k) * ldd + h);
            const float dt = GIVEN ? raw : softplus_(raw + bias);
            dts[k] = dt;
            dAs[k] = GIVEN ? act_load(a_given + (size_t)(tb + k) * ldd + h) : expf(-a * dt);
        }
        __syncthreads();
        for (int k = 0; k < nt; ++k) {
            const float dA = dAs[k], dt = dts[k];
            float xv[CQ], dx[CQ], acc[CQ];
#pragma unroll
            for (int q = 0; q < CQ; ++q) xv[q] = xs[k * CPB + col * CQ + q], dx[q] = dt * xv[q], acc[q] = 0.f;
            decay *= dA;
            const float4 *Bk = reinterpret_cast<const float4 *>(Bs + (size_t)k * NS) + ln, *Ck = reinterpret_cast<const float4 *>(Cs + (size_t)k * NS) + ln;
#pragma unroll
            for (int j = 0; j < RN / 4; ++j) {
                const float4 b = Bk[j * LN];
#pragma unroll
                for (int q = 0; q < CQ; ++q) {
                    S[q][4 * j] = fmaf(dA, S[q][4 * j], dx[q] * b.x), S[q][4 * j + 1] = fmaf(dA, S[q][4 * j + 1], dx[q] * b.y);
                    S[q][4 * j + 2] = fmaf(dA, S[q][4 * j + 2], dx[q] * b.z), S[q][4 * j + 3] = fmaf(dA, S[q][4 * j + 3], dx[q] * b.w);
                }
                if (want_y) {
                    const float4 c = Ck[j * LN];
#pragma unroll
                    for (int q = 0; q < CQ; ++q) {
                        acc[q] = fmaf(S[q][4 * j], c.x, acc[q]), acc[q] = fmaf(S[q][4 * j + 1], c.y, acc[q]);
                        acc[q] = fmaf(S[q][4 * j + 2], c.z, acc[q]), acc[q] = fmaf(S[q][4 * j + 3], c.w, acc[q]);
                    }
                }
            }
            if (want_y) {
#pragma unroll
                for (int q = 0; q < CQ; ++q) {
                    for (int o = LN >> 1; o > 0; o >>= 1) acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], o);
                    if (ln == 0 && p0 + q < P) y[(size_t)(tb + k) * ldy + (size_t)h * P + p0 + q] = fmaf(dsk, xv[q], acc[q]);
                }
            }
        }
    }
#pragma unroll
    for (int q = 0; q < CQ; ++q)
        if (p0 + q < P) {
#pragma unroll
            for (int i = 0; i < RN; i += 4) {
                float *at = st + (size_t)(p0 + q) * N + n_of(i);
                if (QUADS) {
                    if (n_of(i) < N) *reinterpret_cast<float4 *>(at) = make_float4(S[q][i], S[q][i + 1], S[q][i + 2], S[q][i + 3]);
                } else {
#pragma unroll
                    for (int e = 0; e < 4; ++e)
                        if (n_of(i) + e < N) at[e] = S[q][i + e];
                }
            }
        }
    if (decay_out != nullptr && blockIdx.x == 0 && tid == 0) decay_out[(size_t)s * Hs + h] = decay;
}

// The chain over a request's pieces: scratch[c] holds what piece c's scan from zero left; it becomes the state piece c
// starts from, S_start(c + 1) = decay(c) S_start(c) + left(c); the request's slot gives the first start and takes the
// last end.  One thread per float of the state, the pieces of a request in order.
__global__ void __launch_bounds__(256) ssd_chain_kernel(float *__restrict__ scratch, long long scratch_ld, const float *__restrict__ decay,
                                                        float *__restrict__ state, long long state_ld, const int *__restrict__ first_piece,
                                                        const int *__restrict__ slots, int Hs, int PN) {
    pdl_trigger();
    pdl_wait();
    const int s = blockIdx.y;
    const int i = blockIdx.x * 256 + threadIdx.x;
    if (i >= Hs * PN) return;
    const int h = i / PN;
    float *st = state + (size_t)slots[s] * state_ld + i;
    float S = act_load(st);
    const int c0 = first_piece[s], c1 = first_piece[s + 1];
    constexpr int AHEAD = 8;            // the loads of eight pieces are in flight before the first is used
    for (int c = c0; c < c1; c += AHEAD) {
        float left[AHEAD], d[AHEAD];
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c + u < c1) left[u] = act_load(scratch + (size_t)(c + u) * scratch_ld + i), d[u] = act_load(decay + (size_t)(c + u) * Hs + h);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u)
            if (c + u < c1) {
                scratch[(size_t)(c + u) * scratch_ld + i] = S;
                S = fmaf(d[u], S, left[u]);
            }
    }
    *st = S;
}

// ---- a long portion in chunks of 64 tokens, as matrix products ------------------------------------------------
// With G_i the sum of a chunk's log decays up to token i (in double precision, so that a difference keeps float32's) and S0 the state
// ahead of the chunk:
//
//   left behind  e^(G_last) S0 + sum_j e^(G_last - G_j) dt_j x_j B_j^T
//   y_i          e^(G_i) S0 C_i + sum_(j <= i) e^(G_i - G_j) dt_j (C_i . B_j) x_j + D x_i
//
// The first kernel gives what every chunk leaves from a zero state, ssd_chain_kernel the state each starts from, the second kernel y: the
// chunks side by side.  The products go through the tensor cores with both operands in three parts that hold all their bits
// (bf16_thirds.cuh).  Bound by what a block waits for between its few products (two blocks an SM); 32 heads of 64 columns by 128 entries, scans of
// every chunk from zero and from its start, and now: 1,012 tokens in two requests 208 and 73 us, 2,048 tokens 306 and 123 (62 and 102 with
// two tf32 halves, which held 23 bits).  Off 64 bits, y and state, 1,012 tokens: 3.5e-7 and 3.8e-7 the scans, 1.3e-7 and 1.1e-7 here; with decays
// of a few per cent a chunk 3.9e-6 and 5.1e-6, 1.5e-7 and 1.3e-7; of one sign 3.3e-7 and 4.2e-7, 7e-8 and 5e-8; one term in 16 3.7e-7 and
// 6.3e-7, 8e-8 and 1.2e-7.  Numbers below 2^-110 lose what of their parts is below 2^-133.
constexpr int CHUNK = 64, CHUNK_THREADS = 256;
constexpr int CHUNK_N = 128, CHUNK_P = 64;                  // most state entries a column; columns of a block
constexpr int LD_T = 8;                                     // rows that are walked along k: row lengths of 8 over a multiple of 32 put k = 0 .. 3 of
constexpr int LD_B = CHUNK_N + LD_T, LD_X = CHUNK_P + LD_T; // eight neighbouring columns into all banks
constexpr int LD_C = CHUNK_N + 16;                          // rows read 16 bytes a lane, two rows at a time: 16 over
constexpr int LD_M = CHUNK + 4;

struct ChunkArgs {
    const float *xbc;
    int ldx;
    const float *dt_raw;
    int ldd;
    const float *dt_bias, *a_log, *d_skip;
    const int *chunks;              // [n_chunks][2]: first token, past the last
    float *left, *decay;            // [n_chunks][Hs P N], [n_chunks][Hs]
    float *y;
    int ldy, Hs, G, P, N;
};

__device__ __forceinline__ void copy_16(float *dst, const float *src, bool there) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(there ? 16 : 0) : "memory");
}
__device__ __forceinline__ void copies_there() { asm volatile("cp.async.commit_group;\n\tcp.async.wait_group 0;" ::: "memory"); }

// dt and the sums of the log decays of a chunk's tokens (0 behind the last), by one warp
__device__ __forceinline__ void chunk_decays(const ChunkArgs &p, int h, int t0, int nt, float *dts, double *Gs) {
    const int lane = threadIdx.x & 31;
    const float a = expf(__ldg(p.a_log + h)), bias = __ldg(p.dt_bias + h);
    double l[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
        const int i = 2 * lane + u;
        const float dt = i < nt ? softplus_(act_load(p.dt_raw + (size_t)(t0 + i) * p.ldd + h) + bias) : 0.f;
        dts[i] = dt;
        // (a decay below e^-104 is 0 in float32: nothing is kept.  No lower than e^-200 here, or sums of infinite logarithms would have no
        // differences: heads with a_log of 88 and more, whose a dt is infinite.  A NaN stays one.)
        const double log_decay = i < nt ? -(double)(a * dt) : 0.0;
        l[u] = log_decay < -200.0 ? -200.0 : log_decay;
    }
    double sum = l[0] + l[1];
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const double up = __shfl_up_sync(0xffffffffu, sum, o);
        if (lane >= o) sum += up;
    }
    Gs[2 * lane] = sum - l[1], Gs[2 * lane + 1] = sum;
}

// A block with a result that is no finite number goes through its chunk again token by token, as the scan above does, and such results
// come from there: an infinity is lost between the parts of a product, or meets the zero of an earlier row.  A thread owns up to 32 entries of a column.
// OUT: y, from the state S0 (else what is left, from zero).
template <bool OUT>
__device__ __noinline__ void scan_again(const ChunkArgs &p, int c, int h, int col0, int cols, int t0, int nt, const float *Xs, const float *dts, const float *Bs,
                                        const float *Cs, const float *S0) {
    const int col = threadIdx.x >> 2, part = threadIdx.x & 3;
    const float a = expf(__ldg(p.a_log + h)), skip = OUT ? __ldg(p.d_skip + h) : 0.f;
    const float *B = p.xbc + (size_t)t0 * p.ldx + p.Hs * p.P + (h / (p.Hs / p.G)) * p.N;
    float S[CHUNK_N / 4];
#pragma unroll
    for (int i = 0; i < CHUNK_N / 4; ++i) S[i] = OUT ? S0[col * LD_C + (i >> 2) * 16 + part * 4 + (i & 3)] : 0.f;
#pragma unroll 1
    for (int t = 0; t < nt; ++t) {
        const float x = Xs[t * LD_X + col], dA = expf(-a * dts[t]), dx = dts[t] * x;
        float acc = 0.f;
#pragma unroll
        for (int i = 0; i < CHUNK_N / 16; ++i) {
            const int n = i * 16 + part * 4;
            if (n >= p.N) continue;
            const float4 b = OUT ? act_load(reinterpret_cast<const float4 *>(B + (size_t)t * p.ldx + n)) : *reinterpret_cast<const float4 *>(Bs + t * LD_B + n);
            S[4 * i] = fmaf(dA, S[4 * i], dx * b.x), S[4 * i + 1] = fmaf(dA, S[4 * i + 1], dx * b.y);
            S[4 * i + 2] = fmaf(dA, S[4 * i + 2], dx * b.z), S[4 * i + 3] = fmaf(dA, S[4 * i + 3], dx * b.w);
            if (OUT) {
                const float4 v = *reinterpret_cast<const float4 *>(Cs + t * LD_C + n);
                acc = fmaf(S[4 * i], v.x, acc), acc = fmaf(S[4 * i + 1], v.y, acc), acc = fmaf(S[4 * i + 2], v.z, acc), acc = fmaf(S[4 * i + 3], v.w, acc);
            }
        }
        if (OUT) {
            acc += __shfl_xor_sync(0xffffffffu, acc, 1);
            acc += __shfl_xor_sync(0xffffffffu, acc, 2);
            float *y = p.y + (size_t)(t0 + t) * p.ldy + (size_t)h * p.P + col0 + col;
            if (part == 0 && col < cols && !isfinite(act_load(y))) *y = fmaf(skip, x, acc);
        }
    }
    if (!OUT && col < cols) {
        float *left = p.left + ((size_t)c * p.Hs + h) * p.P * p.N + (size_t)(col0 + col) * p.N;
#pragma unroll
        for (int i = 0; i < CHUNK_N / 4; ++i) {
            const int n = (i >> 2) * 16 + part * 4 + (i & 3);
            if (n < p.N && !isfinite(act_load(left + n))) left[n] = S[i];
        }
    }
}

// Block: (chunk, head, 64 columns).  A warp has 32 state entries of 32 columns.
__global__ void __launch_bounds__(CHUNK_THREADS) ssd_chunk_left_kernel(const ChunkArgs p) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    float *Bs = sm, *Xs = Bs + CHUNK * LD_B;
    __shared__ float dts[CHUNK], fs[CHUNK];
    __shared__ double Gs[CHUNK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int c = blockIdx.x, h = blockIdx.y, col0 = blockIdx.z * CHUNK_P, cols = min(CHUNK_P, p.P - col0);
    const int t0 = p.chunks[2 * c], nt = min(p.chunks[2 * c + 1] - t0, CHUNK);
    const float *B = p.xbc + (size_t)t0 * p.ldx + p.Hs * p.P + (h / (p.Hs / p.G)) * p.N, *X = p.xbc + (size_t)t0 * p.ldx + h * p.P + col0;
    for (int i = tid; i < CHUNK * (CHUNK_N / 4); i += CHUNK_THREADS) {
        const int r = i / (CHUNK_N / 4), n = i % (CHUNK_N / 4) * 4;
        const bool there = r < nt && n < p.N;
        copy_16(Bs + r * LD_B + n, there ? B + (size_t)r * p.ldx + n : B, there);
    }
    for (int i = tid; i < CHUNK * (CHUNK_P / 4); i += CHUNK_THREADS) {
        const int r = i / (CHUNK_P / 4), x = i % (CHUNK_P / 4) * 4;
        const bool there = r < nt && x < cols;
        copy_16(Xs + r * LD_X + x, there ? X + (size_t)r * p.ldx + x : X, there);
    }
    if (warp == 0) {
        chunk_decays(p, h, t0, nt, dts, Gs);
        __syncwarp();
        for (int i = lane; i < CHUNK; i += 32) fs[i] = expf((float)(Gs[CHUNK - 1] - Gs[i])) * dts[i];
        if (blockIdx.z == 0 && lane == 0) p.decay[(size_t)c * p.Hs + h] = expf((float)Gs[CHUNK - 1]);
    }
    copies_there();
    __syncthreads();
    const int n0 = (warp & 3) * 32, x0 = (warp >> 2) * 32;
    bool again = false;
    if (n0 < p.N && x0 < cols) {
        float sum[2][4][4] = {};
#pragma unroll 1
        for (int k0 = 0; k0 < nt; k0 += 16) {
            float w[2][2][4], a[4][4];
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const float *bk = Bs + (k0 + 4 * s + q) * LD_B + n0 + g, *xk = Xs + (k0 + 4 * s + q) * LD_X + x0 + g, f = fs[k0 + 4 * s + q];
#pragma unroll
                for (int i = 0; i < 4; ++i) w[i >> 1][i & 1][s] = bk[8 * i], a[i][s] = xk[8 * i] * f;
            }
            float4 wv[2][2], av[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                wv[i >> 1][i & 1] = make_float4(w[i >> 1][i & 1][0], w[i >> 1][i & 1][1], w[i >> 1][i & 1][2], w[i >> 1][i & 1][3]);
                av[i] = make_float4(a[i][0], a[i][1], a[i][2], a[i][3]);
            }
            add_run<2, 4>(sum, wv, av);
        }
        float *out = p.left + ((size_t)c * p.Hs + h) * p.P * p.N + (size_t)col0 * p.N;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const int n = n0 + i * 16 + (e >> 1) * 8 + g, x = x0 + j * 8 + q * 2 + (e & 1);
                    if (n < p.N && x < cols) {
                        out[(size_t)x * p.N + n] = sum[i][j][e];
                        again |= !isfinite(sum[i][j][e]);
                    }
                }
    }
    if (__syncthreads_or(again)) scan_again<false>(p, c, h, col0, cols, t0, nt, Xs, dts, Bs, nullptr, nullptr);
}

// Block: (chunk, `heads` heads of a group, 64 columns).  A warp has 16 tokens (four runs of them) and half of the columns; C B^T, the same for all
// heads of a group, stays in its registers.
constexpr size_t CHUNK_OUT_SMEM = sizeof(float) * (2 * CHUNK * LD_C + CHUNK * LD_X + CHUNK * LD_M);
constexpr size_t CHUNK_LEFT_SMEM = sizeof(float) * CHUNK * (LD_B + LD_X);

__global__ void __launch_bounds__(CHUNK_THREADS, 2) ssd_chunk_out_kernel(const ChunkArgs p, int heads) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ __align__(16) float sm[];
    float *Cs = sm, *BS = Cs + CHUNK * LD_C, *Xs = BS + CHUNK * LD_C, *Ms = Xs + CHUNK * LD_X;       // BS: B, then a head's state
    __shared__ float dts[CHUNK];
    __shared__ double Gs[CHUNK];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int c = blockIdx.x, h0 = blockIdx.y * heads, col0 = blockIdx.z * CHUNK_P, cols = min(CHUNK_P, p.P - col0);
    const int t0 = p.chunks[2 * c], nt = min(p.chunks[2 * c + 1] - t0, CHUNK), kn = (p.N + 15) / 16 * 16;
    const float *B = p.xbc + (size_t)t0 * p.ldx + p.Hs * p.P + (h0 / (p.Hs / p.G)) * p.N, *C = B + p.G * p.N;
    for (int i = tid; i < CHUNK * (CHUNK_N / 4); i += CHUNK_THREADS) {
        const int r = i / (CHUNK_N / 4), n = i % (CHUNK_N / 4) * 4;
        const bool there = r < nt && n < p.N;
        copy_16(BS + r * LD_C + n, there ? B + (size_t)r * p.ldx + n : B, there);
        copy_16(Cs + r * LD_C + n, there ? C + (size_t)r * p.ldx + n : C, there);
    }
    copies_there();
    __syncthreads();
    const int i0 = (warp & 3) * 16, x0 = (warp >> 2) * 32;           // this warp's tokens, and its columns (of C B^T: earlier tokens)
    float cb[1][4][4] = {};
    if (x0 <= i0 + 15) {
        for (int k = 0; k < kn; k += 16) {
            float4 w[1][2], a[4];
            w[0][0] = *reinterpret_cast<const float4 *>(Cs + (i0 + g) * LD_C + k + 4 * q);
            w[0][1] = *reinterpret_cast<const float4 *>(Cs + (i0 + 8 + g) * LD_C + k + 4 * q);
#pragma unroll
            for (int j = 0; j < 4; ++j) a[j] = *reinterpret_cast<const float4 *>(BS + (x0 + j * 8 + g) * LD_C + k + 4 * q);
            add_run<1, 4>(cb, w, a);
        }
    }
    for (int h = h0; h < h0 + heads; ++h) {
        __syncthreads();                                             // the head before is done with BS, Xs, Ms and its decays
        const float *S0 = p.left + ((size_t)c * p.Hs + h) * p.P * p.N + (size_t)col0 * p.N, *X = p.xbc + (size_t)t0 * p.ldx + h * p.P + col0;
        for (int i = tid; i < CHUNK_P * (CHUNK_N / 4); i += CHUNK_THREADS) {
            const int r = i / (CHUNK_N / 4), n = i % (CHUNK_N / 4) * 4;
            const bool there = r < cols && n < p.N;
            copy_16(BS + r * LD_C + n, there ? S0 + (size_t)r * p.N + n : S0, there);
        }
        for (int i = tid; i < CHUNK * (CHUNK_P / 4); i += CHUNK_THREADS) {
            const int r = i / (CHUNK_P / 4), x = i % (CHUNK_P / 4) * 4;
            const bool there = r < nt && x < cols;
            copy_16(Xs + r * LD_X + x, there ? X + (size_t)r * p.ldx + x : X, there);
        }
        if (warp == 0) chunk_decays(p, h, t0, nt, dts, Gs);
        __syncthreads();
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                const int i = i0 + (e >> 1) * 8 + g, t = x0 + j * 8 + q * 2 + (e & 1);
                Ms[i * LD_M + t] = t <= i ? cb[0][j][e] * (expf((float)(Gs[i] - Gs[t])) * dts[t]) : 0.f;
            }
        copies_there();
        __syncthreads();
        bool again = false;
        if (x0 < cols && i0 < nt) {
            float old[1][4][4] = {}, now[1][4][4] = {};
            for (int k = 0; k < kn; k += 16) {
                float4 w[1][2], a[4];
                w[0][0] = *reinterpret_cast<const float4 *>(Cs + (i0 + g) * LD_C + k + 4 * q);
                w[0][1] = *reinterpret_cast<const float4 *>(Cs + (i0 + 8 + g) * LD_C + k + 4 * q);
#pragma unroll
                for (int j = 0; j < 4; ++j) a[j] = *reinterpret_cast<const float4 *>(BS + (x0 + j * 8 + g) * LD_C + k + 4 * q);
                add_run<1, 4>(old, w, a);
            }
            for (int k = 0; k <= i0; k += 16) {                      // tokens behind this warp's last have no part
                float w[2][4], a[4][4];
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const int t = k + 4 * s + q;
                    w[0][s] = Ms[(i0 + g) * LD_M + t], w[1][s] = Ms[(i0 + 8 + g) * LD_M + t];
#pragma unroll
                    for (int j = 0; j < 4; ++j) a[j][s] = Xs[t * LD_X + x0 + j * 8 + g];
                }
                float4 wv[1][2], av[4];
                wv[0][0] = make_float4(w[0][0], w[0][1], w[0][2], w[0][3]), wv[0][1] = make_float4(w[1][0], w[1][1], w[1][2], w[1][3]);
#pragma unroll
                for (int j = 0; j < 4; ++j) av[j] = make_float4(a[j][0], a[j][1], a[j][2], a[j][3]);
                add_run<1, 4>(now, wv, av);
            }
            const float skip = __ldg(p.d_skip + h);
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const int i = i0 + r * 8 + g;
                const float kept = expf((float)Gs[i]);
                if (i < nt) {
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int x = x0 + j * 8 + q * 2;
                        if (x >= cols) continue;
                        const float2 xv = *reinterpret_cast<const float2 *>(Xs + i * LD_X + x);
                        float2 v = make_float2(fmaf(kept, old[0][j][2 * r], now[0][j][2 * r]), fmaf(kept, old[0][j][2 * r + 1], now[0][j][2 * r + 1]));
                        v = make_float2(fmaf(skip, xv.x, v.x), fmaf(skip, xv.y, v.y));
                        again |= !isfinite(v.x) || !isfinite(v.y);
                        *reinterpret_cast<float2 *>(p.y + (size_t)(t0 + i) * p.ldy + (size_t)h * p.P + col0 + x) = v;
                    }
                }
            }
        }
        if (__syncthreads_or(again)) scan_again<true>(p, c, h, col0, cols, t0, nt, Xs, dts, nullptr, Cs, BS);
    }
}

// out[t, c] = (y[t, c] silu(z[t, c])) / rms over c's part * w[c]; block (token, part).  The gated values wait in shared
// memory between the sum of squares and the division when a part fits there (keep != 0): y and z are then read once.
template <typename TO, int NT>
__global__ void __launch_bounds__(NT) ssd_gate_norm_kernel(const float *__restrict__ y, int ldy, const float *__restrict__ z, int ldz,
                                                             const float *__restrict__ w, TO *__restrict__ out, int ldo, int part, float eps, int keep) {
    pdl_trigger();
    pdl_wait();
    extern __shared__ float gated[];
    __shared__ float red[32];
    const int t = blockIdx.x, c0 = blockIdx.y * part;
    const float *yr = y + (size_t)t * ldy + c0, *zr = z + (size_t)t * ldz + c0;
    float ss = 0.f;
#pragma unroll 4
    for (int i = threadIdx.x; i < part; i += NT) {
        const float v = act_load(yr + i) * silu_(act_load(zr + i));
        if (keep) gated[i] = v;
        ss = fmaf(v, v, ss);
    }
    const float inv = 1.0f / sqrtf(block_sum(ss, red) / (float)part + eps);
    TO *orow = out + (size_t)t * ldo + c0;
#pragma unroll 4
    for (int i = threadIdx.x; i < part; i += NT) {
        const float v = keep ? gated[i] : act_load(yr + i) * silu_(act_load(zr + i));
        orow[i] = from_f32<TO>(v * inv * __ldg(w + c0 + i));
    }
}

}  // namespace

namespace {
int scan_any(const float *xbc, int ldx, const float *dt_raw, int ldd, const float *dt_bias, const float *a_log, const float *d_skip,
                           float *state, long long state_ld, const int *seq_start, const int *slots, float *y, int ldy, int n_seqs, int Hs, int G,
                           int P, int N, int pieces, int zero_start, float *decay_out, const float *a_given, int Px, int max_tokens, cudaStream_t stream) {
    LGML_REQUIRE(n_seqs >= 0 && Hs > 0 && G > 0 && P > 0 && N > 0 && Px > 0 && Px <= P, "ssd_scan: bad sizes");
    LGML_REQUIRE(Hs % G == 0, "ssd_scan: %d heads are no multiple of %d groups", Hs, G);
    LGML_REQUIRE(N <= 1024, "ssd_scan: a state of %d numbers per column is more than 1024", N);
    LGML_REQUIRE(state_ld >= (long long)Hs * P * N, "ssd_scan: the state's rows do not hold %d x %d x %d floats", Hs, P, N);
    LGML_REQUIRE(ldx >= Hs * Px + 2 * G * N && ldd >= Hs && ldy >= Hs * P, "ssd_scan: rows too short");
    LGML_REQUIRE(n_seqs <= 65535 && Hs <= 65535, "ssd_scan: too many requests, pieces or heads");
    LGML_REQUIRE(slots != nullptr || pieces, "ssd_scan: requests come with their slots");
    if (n_seqs == 0) return 0;
    // RN entries a lane, LN lanes a column (a power of two up to 32): the pair that wastes least, then the smaller RN.
    // Up to 16 entries a lane for states of up to 512 numbers a column (four columns a thread then have registers), else up to 32.
    const bool quad = N <= 512;
    static const int rns[6] = {4, 8, 12, 16, 24, 32};
    int best_rn = 32, best_ln = 32, best_cover = 1 << 30;
    for (int i = 0; i < 6; ++i) {
        if (quad ? rns[i] > 16 : rns[i] < 8) continue;
        int ln = 1;
        while (ln * rns[i] < N && ln < 32) ln *= 2;
        if (ln * rns[i] < N) continue;
        // (at equal cover: with four columns a thread the larger RN, fewer lanes to add up; with one the smaller, more threads)
        if (ln * rns[i] < best_cover || (quad && ln * rns[i] == best_cover)) best_cover = ln * rns[i], best_rn = rns[i], best_ln = ln;
    }
    // One column a thread (the same sums) up to 512 blocks of four columns a thread: more blocks for SMs without one, and shorter chains.  32 heads of
    // 64 columns by 128 entries, microseconds, four columns with the state element by element; four with 16 bytes at a time; one: 2 requests
    // of one token 6.5, 4.1, 3.7; 8 9.0, 6.5, 6.8; 32 24.4, 17.1, 18.5; 2 of 100 tokens 76, 82, 51; 16 of 100 195, 198, 179; 32 of 16 62, 59, 65.
    const long long wide_blocks = (long long)((P + SCAN_THREADS / best_ln * 4 - 1) / (SCAN_THREADS / best_ln * 4)) * Hs * n_seqs;
    const bool four = quad && wide_blocks > 512;
    const int LN = best_ln, CQ = four ? 4 : 1, CPB = (SCAN_THREADS / LN) * CQ;
    const int NS = LN * best_rn;
    int TT = 32;
    while (TT > 1 && (size_t)TT * (2 * NS + CPB + 2) * sizeof(float) > 46 * 1024) TT /= 2;
    const size_t smem = (size_t)TT * (2 * NS + CPB + 2) * sizeof(float);
    dim3 grid((P + CPB - 1) / CPB, Hs, n_seqs);
    const int vec = N % 4 == 0 && ldx % 4 == 0 && (Hs * Px) % 4 == 0 && ((uintptr_t)xbc & 15) == 0;
#define LGML_SCAN_Q(RN, CQ, GIVEN, QUADS) lgml_launch(ssd_scan_kernel<RN, CQ, GIVEN, QUADS>, grid, SCAN_THREADS, smem, stream, xbc, ldx, dt_raw, ldd, dt_bias, a_log, d_skip, \
                                               state, state_ld, seq_start, slots, y, ldy, Hs, G, P, N, LN, TT, pieces, zero_start, decay_out, vec, a_given, Px, max_tokens)
#define LGML_SCAN_K(RN, CQ, GIVEN) do { if (quads) LGML_SCAN_Q(RN, CQ, GIVEN, true); else LGML_SCAN_Q(RN, CQ, GIVEN, false); } while (0)
#define LGML_SCAN(RN, CQ) do { if (a_given != nullptr) LGML_SCAN_K(RN, CQ, true); else LGML_SCAN_K(RN, CQ, false); } while (0)
    const bool quads = N % 4 == 0 && state_ld % 4 == 0 && ((uintptr_t)state & 15) == 0;
    if (four) {
        switch (best_rn) {
            case 4: LGML_SCAN(4, 4); break;
            case 8: LGML_SCAN(8, 4); break;
            case 12: LGML_SCAN(12, 4); break;
            default: LGML_SCAN(16, 4); break;
        }
    } else {
        switch (best_rn) {
            case 4: LGML_SCAN(4, 1); break;
            case 8: LGML_SCAN(8, 1); break;
            case 12: LGML_SCAN(12, 1); break;
            case 16: LGML_SCAN(16, 1); break;
            case 24: LGML_SCAN(24, 1); break;
            default: LGML_SCAN(32, 1); break;
        }
    }
#undef LGML_SCAN
#undef LGML_SCAN_K
#undef LGML_SCAN_Q
    return lgml_launch_status("ssd_scan");
}
}  // namespace

LGML_API int lgml_ssd_scan(const float *xbc, int ldx, const float *dt_raw, int ldd, const float *dt_bias, const float *a_log, const float *d_skip,
                           float *state, long long state_ld, const int *seq_start, const int *slots, float *y, int ldy, int n_seqs, int Hs, int G,
                           int P, int N, int pieces, int zero_start, float *decay_out, cudaStream_t stream) {
    return scan_any(xbc, ldx, dt_raw, ldd, dt_bias, a_log, d_skip, state, state_ld, seq_start, slots, y, ldy, n_seqs, Hs, G, P, N, pieces, zero_start,
                    decay_out, nullptr, P, 0, stream);
}

// The recurrence with decays and write weights given: decay / weight float32 rows of Hs entries, ldd apart.  x has Px columns per head,
// the state and y have P >= Px; columns from Px on are written with x = 1.  max_tokens > 0: requests that bring more
// tokens are left out.
LGML_API int lgml_ssd_scan_given(const float *xbc, int ldx, const float *weight, const float *decay, int ldd, float *state, long long state_ld,
                                 const int *seq_start, const int *slots, float *y, int ldy, int n_seqs, int Hs, int G, int Px, int P, int N, int pieces,
                                 int zero_start, float *decay_out, int max_tokens, cudaStream_t stream) {
    LGML_REQUIRE(max_tokens == 0 || !pieces, "ssd_scan: pieces leave no request out");
    LGML_REQUIRE(decay != nullptr && weight != nullptr, "ssd_scan: decays and write weights are missing");
    return scan_any(xbc, ldx, weight, ldd, nullptr, nullptr, nullptr, state, state_ld, seq_start, slots, y, ldy, n_seqs, Hs, G, P, N, pieces, zero_start,
                    decay_out, decay, Px, max_tokens, stream);
}

LGML_API int lgml_ssd_gate_norm(const float *y, int ldy, const float *z, int ldz, const float *w, void *out, int out_dtype, int ldo, int n_tokens,
                                int inner, int groups, float eps, cudaStream_t stream) {
    LGML_REQUIRE(n_tokens >= 0 && inner > 0 && groups > 0 && inner % groups == 0, "ssd_gate_norm: %d channels in %d parts", inner, groups);
    LGML_REQUIRE(ldy >= inner && ldz >= inner && ldo >= inner && groups <= 65535, "ssd_gate_norm: rows too short");
    if (n_tokens == 0) return 0;
    dim3 grid(n_tokens, groups);
    const int part = inner / groups;
    const int threads = (n_tokens * groups <= 296 && part >= 1024) ? 1024 : 256;      // few rows: more threads share a row's latency
    const int keep = (size_t)part * sizeof(float) <= 40 * 1024;
    const size_t smem = keep ? (size_t)part * sizeof(float) : 0;
#define LGML_GN(TO, NT) lgml_launch(ssd_gate_norm_kernel<TO, NT>, grid, NT, smem, stream, y, ldy, z, ldz, w, (TO *)out, ldo, part, eps, keep)
    if (out_dtype == LGML_F32) { if (threads == 1024) LGML_GN(float, 1024); else LGML_GN(float, 256); }
    else if (out_dtype == LGML_BF16) { if (threads == 1024) LGML_GN(__nv_bfloat16, 1024); else LGML_GN(__nv_bfloat16, 256); }
    else LGML_FAIL("ssd_gate_norm: unknown output type %d", out_dtype);
#undef LGML_GN
    return lgml_launch_status("ssd_gate_norm");
}

// See ssd_chain_kernel.  scratch: [pieces, >= Hs P N]; decay: [pieces, Hs]; first_piece: [n_seqs + 1].
LGML_API int lgml_ssd_chain(float *scratch, long long scratch_ld, const float *decay, float *state, long long state_ld, const int *first_piece,
                            const int *slots, int n_seqs, int Hs, int P, int N, cudaStream_t stream) {
    LGML_REQUIRE(n_seqs >= 0 && Hs > 0 && P > 0 && N > 0 && n_seqs <= 65535, "ssd_chain: bad sizes");
    LGML_REQUIRE(scratch_ld >= (long long)Hs * P * N && state_ld >= (long long)Hs * P * N, "ssd_chain: rows too short");
    if (n_seqs == 0) return 0;
    dim3 grid((Hs * P * N + 255) / 256, n_seqs);
    lgml_launch(ssd_chain_kernel, grid, 256, 0, stream, scratch, scratch_ld, decay, state, state_ld, first_piece, slots, Hs, P * N);
    return lgml_launch_status("ssd_chain");
}

// A portion in chunks of 64 tokens: what every chunk leaves from a zero state (y null), or y from the states that ssd_chain made of it.  `left`: [n_chunks, Hs P N],
// 16-byte aligned; N a multiple of 4 up to 128, P a multiple of 4, rows of xbc on 16 bytes.
LGML_API int lgml_ssd_chunks(const float *xbc, int ldx, const float *dt_raw, int ldd, const float *dt_bias, const float *a_log, const float *d_skip,
                             const int *chunks, int n_chunks, float *left, float *decay, float *y, int ldy, int Hs, int G, int P, int N, cudaStream_t stream) {
    LGML_REQUIRE(n_chunks >= 0 && Hs > 0 && G > 0 && P > 0 && N > 0 && Hs % G == 0 && Hs <= 65535, "ssd_chunks: bad sizes");
    LGML_REQUIRE(N % 4 == 0 && N <= CHUNK_N && P % 4 == 0 && ldx % 4 == 0 && (((uintptr_t)xbc | (uintptr_t)left) & 15) == 0, "ssd_chunks: sizes or rows it does not take");
    LGML_REQUIRE(ldx >= Hs * P + 2 * G * N && ldd >= Hs, "ssd_chunks: rows too short");
    LGML_REQUIRE(y == nullptr || (ldy >= Hs * P && ldy % 2 == 0 && ((uintptr_t)y & 7) == 0), "ssd_chunks: rows too short or not aligned");
    if (n_chunks == 0) return 0;
    const ChunkArgs p = {xbc, ldx, dt_raw, ldd, dt_bias, a_log, d_skip, chunks, left, decay, y, ldy, Hs, G, P, N};
    const int tiles = (P + CHUNK_P - 1) / CHUNK_P;
    auto kernel_smem = [](const void *kernel, size_t smem) { return cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); };
    if (y == nullptr) {
        if (kernel_smem((const void *)ssd_chunk_left_kernel, CHUNK_LEFT_SMEM) != cudaSuccess) return lgml_launch_status("ssd_chunks");
        lgml_launch(ssd_chunk_left_kernel, dim3(n_chunks, Hs, tiles), CHUNK_THREADS, CHUNK_LEFT_SMEM, stream, p);
    } else {
        if (kernel_smem((const void *)ssd_chunk_out_kernel, CHUNK_OUT_SMEM) != cudaSuccess) return lgml_launch_status("ssd_chunks");
        // As many heads a block as leave nearly two blocks an SM (32 heads, 1, 2 and 4 a block, all three kernels: 129 tokens 27, 34 and 50 us,
        // 488 tokens 40, 43 and 57, 1,012 tokens 72, 65 and 85, 2,048 tokens 118, 111 and 105).
        int heads = 4;
        while (heads > 1 && ((Hs / G) % heads || (long long)n_chunks * tiles * (Hs / heads) < 252)) heads /= 2;
        lgml_launch(ssd_chunk_out_kernel, dim3(n_chunks, Hs / heads, tiles), CHUNK_THREADS, CHUNK_OUT_SMEM, stream, p, heads);
    }
    return lgml_launch_status("ssd_chunks");
}
