// The delta rule with a decay per key channel (delta_rule.cu) over many tokens, eight at a time.
//
// Token by token every step waits for two sums over a column of S, each ending in shuffles: 0.34 us a
// token, whatever the chip has free.  Over eight tokens from S0, with G_i the decays' product of the
// block's tokens 0 .. i and G_ji that of tokens j + 1 .. i (element by element over the key's entries):
//     p_i = (G_i k_i)^T S0        u_i = beta_i (v_i - p_i - sum_{j<i} c_ij u_j),  c_ij = k_i^T (G_ji k_j)
//     o_i = (G_i q_i)^T S0 + sum_{j<=i} d_ij u_j,                                 d_ij = q_i^T (G_ji k_j)
//     S8  = G_7 S0 + sum_j (G_j7 k_j) u_j
// All products of decays run forward in time (no quotients, so decays of any size, zero included, are
// fine), everything is float32, and u is found by forward substitution: what the token-by-token form
// computes, with its sums in another order.  p and the first part of o of all eight tokens are
// independent of each other, so one block pays the latency that one token did.
//
//   delta_block_prepare   per (block, head), a warp: the decayed vectors G_i k_i, G_i q_i, G_j7 k_j, G_7, and c, d
//   delta_block_scan      per (request, head, 16 columns): the blocks in order, S in registers.
#include "common.cuh"

LGML_DEFINE_LAST_ERROR(lgml_delta_block)

namespace {
constexpr int L = 8;                     // tokens of a block
constexpr int THREADS = 128, COLS = THREADS / L;     // columns of a CTA of the scan
constexpr int STAGES = 3;

// floats of a block's record: G_i k_i [8, D], G_i q_i [8, D], G_j7 k_j [8, D], G_7 [D], c [8, 8], d [8, 8], beta [8]
__host__ __device__ constexpr int record_floats(int D) { return 25 * D + 2 * L * L + L; }

__device__ __forceinline__ void cp_async_16(float *dst, const float *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

__device__ __forceinline__ float4 mul4(float4 a, float4 b) { return make_float4(a.x * b.x, a.y * b.y, a.z * b.z, a.w * b.w); }
__device__ __forceinline__ float dot4(float4 a, float4 b) { return fmaf(a.x, b.x, a.y * b.y) + fmaf(a.z, b.z, a.w * b.w); }

// A warp per (block, head), four of the key's entries a lane (D <= 128).  qkv_c and gb as delta_prepare writes them.
__global__ void __launch_bounds__(THREADS) delta_block_prepare_kernel(const float *__restrict__ qkv_c, const float *__restrict__ gb,
                                                                      const int *__restrict__ rows, float *__restrict__ records, int n_blocks, int C,
                                                                      int H, int G, int D) {
    pdl_trigger();
    pdl_wait();
    const int lane = threadIdx.x & 31;
    const long long unit = (long long)blockIdx.x * (THREADS / 32) + (threadIdx.x >> 5);
    if (unit >= (long long)n_blocks * H) return;
    const int b = (int)(unit / H), h = (int)(unit - (long long)b * H), g = h / (H / G);
    const int t0 = act_load(rows + 2 * b), n = act_load(rows + 2 * b + 1) - t0;
    const int d = lane * 4;
    const bool in = d < D;
    float *rec = records + (size_t)unit * record_floats(D);
    float4 q[L], k[L], dec[L];
#pragma unroll
    for (int i = 0; i < L; ++i) {
        q[i] = k[i] = make_float4(0.f, 0.f, 0.f, 0.f), dec[i] = make_float4(1.f, 1.f, 1.f, 1.f);
        if (in && i < n) {                  // (a token that is not there decays nothing and writes nothing)
            const float *row = qkv_c + (size_t)(t0 + i) * C + g * D + d;
            q[i] = act_load(reinterpret_cast<const float4 *>(row));
            k[i] = act_load(reinterpret_cast<const float4 *>(row + G * D));
            dec[i] = act_load(reinterpret_cast<const float4 *>(gb + ((size_t)(t0 + i) * H + h) * (D + 4) + d));
        }
    }
    if (lane < L) rec[25 * D + 2 * L * L + lane] = lane < n ? act_load(gb + ((size_t)(t0 + lane) * H + h) * (D + 4) + D) : 0.f;
    // val[8 i + j]: c_ij for j < i, d_ji for j >= i
    float val[L * L];
    float4 prod = make_float4(1.f, 1.f, 1.f, 1.f), kj[L];
#pragma unroll
    for (int i = 0; i < L; ++i) {
        prod = mul4(prod, dec[i]);
        kj[i] = k[i];
#pragma unroll
        for (int j = 0; j < L; ++j)
            if (j < i) kj[j] = mul4(kj[j], dec[i]);
#pragma unroll
        for (int j = 0; j < L; ++j) {
            if (j < i) val[L * i + j] = dot4(k[i], kj[j]);
            if (j <= i) val[L * j + i] = dot4(q[i], kj[j]);
        }
        if (in) {
            *reinterpret_cast<float4 *>(rec + i * D + d) = mul4(k[i], prod);
            *reinterpret_cast<float4 *>(rec + (L + i) * D + d) = mul4(q[i], prod);
        }
    }
    if (in) {
#pragma unroll
        for (int j = 0; j < L; ++j) *reinterpret_cast<float4 *>(rec + (2 * L + j) * D + d) = kj[j];
        *reinterpret_cast<float4 *>(rec + 3 * L * D + d) = prod;
    }
    // 64 sums over the warp, halved and scattered: lane x ends with entries 2 x and 2 x + 1
#pragma unroll
    for (int half = 32, mask = 16; mask > 0; half >>= 1, mask >>= 1) {
        const bool upper = (lane & mask) != 0;
#pragma unroll
        for (int e = 0; e < half; ++e) {
            const float send = upper ? val[e] : val[e + half], keep = upper ? val[e + half] : val[e];
            val[e] = keep + __shfl_xor_sync(0xffffffffu, send, mask);
        }
    }
    float *c = rec + 25 * D, *dd = c + L * L;
#pragma unroll
    for (int e = 0; e < 2; ++e) {
        const int s = 2 * lane + e, i = s / L, j = s % L;
        c[s] = j < i ? val[e] : 0.f;
        dd[L * j + i] = j >= i ? val[e] : 0.f;
    }
}

__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    uint64_t r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)), "l"(*reinterpret_cast<uint64_t *>(&c)));
    return *reinterpret_cast<float2 *>(&r);
}

// R lanes share a column, four rows of S each (D <= 4 R), and R / 8 columns a lane: a vector of a block is then read once
// by R different lanes for R / 8 columns, without a bank asked twice.  (Eight lanes on sixteen rows of one column read
// the same floats in every column of a warp, which costs shared memory as many cycles as different ones.)
// 512 tokens of sixteen heads of 128 x 128 on one B200: 74 us, about 2,260 cycles a block of eight tokens; a warp a scheduler, stalled
// a third of the time on shuffles and on the chain of the substitution.  Token by token 238 us; 2,048 tokens 289 and 937 us.
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    uint64_t r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(*reinterpret_cast<uint64_t *>(&a)), "l"(*reinterpret_cast<uint64_t *>(&b)));
    return *reinterpret_cast<float2 *>(&r);
}

// Entry e = 8 c + i of a lane's sums is token i ^ i_own of column c ^ c_own: in that order the halving sums over the lanes
// keep their first entries and send their last ones, whichever lane it is, and a lane's own column is its first.
template <int R>
__global__ void __launch_bounds__(THREADS) delta_block_scan_kernel(const float *__restrict__ qkv_c, const float *__restrict__ records,
                                                                   float *__restrict__ state, long long state_stride, const int *__restrict__ rows,
                                                                   const int *__restrict__ first, const int *__restrict__ requests,
                                                                   const int *__restrict__ slots, float *__restrict__ o_out, int H, int G, int D, int Dv) {
    constexpr int NC = R / L, VEC = 4 * R;                      // columns of a lane; a vector in shared memory
    constexpr int STAGE = 25 * VEC + 2 * L * L + L;
    extern __shared__ __align__(16) float sm[];
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, x = lane % R;
    const int i_own = x % L, c_own = x / L;                     // the token and the column that this lane finishes
    const int h = blockIdx.y, col0 = blockIdx.z * COLS + (tid / R) * NC;
    const int C = 2 * G * D + H * Dv;
    const int b0 = act_load(first + blockIdx.x), nb = act_load(first + blockIdx.x + 1) - b0;
    const int t0 = act_load(rows + 2 * b0), t_end = act_load(rows + 2 * (b0 + nb - 1) + 1);
    float *S_base = state + (size_t)slots[requests[blockIdx.x]] * state_stride + (size_t)h * D * Dv;
    const int d4 = D / 4;
    // rows past D: S and the vectors are zero there
    for (int e = tid; e < STAGES * STAGE; e += THREADS) sm[e] = 0.f;
    __syncthreads();
    auto stage = [&](int b) {
        const float *rec = records + ((size_t)(b0 + b) * H + h) * record_floats(D);
        float *dst = sm + (b % STAGES) * STAGE;
        if (x < d4)
            for (int v = tid / R; v < 25; v += THREADS / R) cp_async_16(dst + v * VEC + x * 4, rec + v * D + x * 4);
        if (tid < (2 * L * L + L) / 4) cp_async_16(dst + 25 * VEC + tid * 4, rec + 25 * D + tid * 4);
    };
    const bool has_own = col0 + c_own < Dv;
    const float *v_own = qkv_c + (size_t)(t0 + i_own) * C + 2 * G * D + (size_t)h * Dv + (has_own ? col0 + c_own : 0);
    auto value = [&](int b) { return has_own && b < nb && t0 + b * L + i_own < t_end ? act_load(v_own + (size_t)b * L * C) : 0.f; };
    stage(0);
    cp_async_commit();
    if (nb > 1) stage(1);
    cp_async_commit();
    float2 S[NC][2];
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        float y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = x < d4 && col0 + (c ^ c_own) < Dv ? S_base[(size_t)(x * 4 + j) * Dv + col0 + (c ^ c_own)] : 0.f;
        S[c][0] = make_float2(y[0], y[1]), S[c][1] = make_float2(y[2], y[3]);
    }
    float v_next = value(0);
    for (int b = 0; b < nb; ++b) {
        cp_async_wait<1>();
        __syncthreads();                    // this block's record is there, and nobody reads the one before any more
        if (b + 2 < nb) stage(b + 2);
        cp_async_commit();
        const float v = v_next;
        v_next = value(b + 1);
        const float *buf = sm + (b % STAGES) * STAGE, *vec = buf + x * 4, *tail = buf + 25 * VEC;
        // this lane's share of the sums over S0 for p and o
        float p[R], o[R];
#pragma unroll
        for (int i = 0; i < L; ++i) {
            const float *at = vec + (i ^ i_own) * VEC;
            const float4 kd = *reinterpret_cast<const float4 *>(at), qd = *reinterpret_cast<const float4 *>(at + L * VEC);
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                float2 a = fma2(make_float2(kd.z, kd.w), S[c][1], mul2(make_float2(kd.x, kd.y), S[c][0]));
                p[c * L + i] = a.x + a.y;
                a = fma2(make_float2(qd.z, qd.w), S[c][1], mul2(make_float2(qd.x, qd.y), S[c][0]));
                o[c * L + i] = a.x + a.y;
            }
        }
        // added up over the column's lanes and scattered: a lane ends with its own entry
#pragma unroll
        for (int half = R / 2; half > 0; half >>= 1) {
#pragma unroll
            for (int e = 0; e < half; ++e) {
                p[e] += __shfl_xor_sync(0xffffffffu, p[e + half], half);
                o[e] += __shfl_xor_sync(0xffffffffu, o[e + half], half);
            }
        }
        float cc[L], dd[L];
#pragma unroll
        for (int j = 0; j < L; j += 4) {
            *reinterpret_cast<float4 *>(cc + j) = *reinterpret_cast<const float4 *>(tail + i_own * L + j);
            *reinterpret_cast<float4 *>(dd + j) = *reinterpret_cast<const float4 *>(tail + L * L + i_own * L + j);
        }
        const float beta = tail[2 * L * L + i_own];
        const float4 gl = *reinterpret_cast<const float4 *>(vec + 24 * VEC);
#pragma unroll
        for (int c = 0; c < NC; ++c) S[c][0] = mul2(S[c][0], make_float2(gl.x, gl.y)), S[c][1] = mul2(S[c][1], make_float2(gl.z, gl.w));
        // Forward substitution; each u goes into S as soon as it is known.  A token adds only the u up to its own: those behind
        // it have factors of zero, but zero times an infinite value is not zero, and a token's result must not depend on later
        // ones.  Tokens that are not there have u = 0, whatever S holds, for the same reason.
        const int t = t0 + b * L + i_own;
        const bool there = t < t_end;
        float w = v - p[0], out = o[0];
#pragma unroll
        for (int j = 0; j < L; ++j) {
            const float4 ku = *reinterpret_cast<const float4 *>(vec + (2 * L + j) * VEC);
            const float mine = there ? beta * w : 0.f;
            float own = 0.f;
#pragma unroll
            for (int c = 0; c < NC; ++c) {
                const float u = __shfl_sync(0xffffffffu, mine, (lane & ~(R - 1)) | ((c ^ c_own) * L + j));
                if (c == 0) own = u;
                const float2 uu = make_float2(u, u);
                S[c][0] = fma2(make_float2(ku.x, ku.y), uu, S[c][0]), S[c][1] = fma2(make_float2(ku.z, ku.w), uu, S[c][1]);
            }
            w = fmaf(-cc[j], own, w);
            out = j <= i_own ? fmaf(dd[j], own, out) : out;
        }
        if (has_own && there) o_out[(size_t)t * H * Dv + (size_t)h * Dv + col0 + c_own] = out;
    }
    cp_async_wait<0>();
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        if (x >= d4 || col0 + (c ^ c_own) >= Dv) continue;
        const float y[4] = {S[c][0].x, S[c][0].y, S[c][1].x, S[c][1].y};
#pragma unroll
        for (int j = 0; j < 4; ++j) S_base[(size_t)(x * 4 + j) * Dv + col0 + (c ^ c_own)] = y[j];
    }
}

template <int R>
int launch_scan(const float *qkv_c, const float *records, float *state, long long state_stride, const int *rows, const int *first, const int *requests,
                const int *slots, float *o_out, int n_requests, int H, int G, int D, int Dv, cudaStream_t stream) {
    const size_t smem = sizeof(float) * STAGES * (25 * (size_t)4 * R + 2 * L * L + L);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(delta_block_scan_kernel<R>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) LGML_FAIL("delta_block: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    }
    lgml_launch_alone(delta_block_scan_kernel<R>, dim3(n_requests, H, (Dv + COLS - 1) / COLS), THREADS, smem, stream, qkv_c, records, state, state_stride, rows,
                first, requests, slots, o_out, H, G, D, Dv);
    return lgml_launch_status("delta_block_scan");
}
}  // namespace

LGML_API int lgml_delta_block_tokens(void) { return L; }
LGML_API long long lgml_delta_block_record_floats(int D) { return record_floats(D); }

// qkv_c and gb as delta_prepare writes them; rows int32 [n_blocks, 2]: a block's first token row and the row past its last (at most
// eight), a request's blocks in order; first int32 [n_requests + 1]: its first block; requests int32 [n_requests]: its row of `slots`.
// records: n_blocks * H * record_floats(D) floats of scratch.
LGML_API int lgml_delta_block_scan(const float *qkv_c, const float *gb, float *state, long long state_stride, const int *rows, int n_blocks,
                                   const int *first, const int *requests, int n_requests, const int *slots, float *records, float *o_out, int H, int G,
                                   int D, int Dv, cudaStream_t stream) {
    LGML_REQUIRE(n_requests >= 0 && n_blocks >= 0 && H > 0 && G > 0 && D > 0 && Dv > 0 && H % G == 0 && H <= 65535, "delta_block: bad sizes");
    LGML_REQUIRE(D % 4 == 0 && D <= 128, "delta_block: key size %d is no multiple of 4 up to 128", D);
    LGML_REQUIRE((H * Dv) % 4 == 0 && (((uintptr_t)qkv_c | (uintptr_t)gb | (uintptr_t)records) & 15) == 0, "delta_block: rows must start on 16 bytes");
    if (n_requests == 0 || n_blocks == 0) return 0;
    const int C = 2 * G * D + H * Dv;
    const long long units = (long long)n_blocks * H, blocks = (units + THREADS / 32 - 1) / (THREADS / 32);
    LGML_REQUIRE(blocks <= 0x7fffffffLL, "delta_block: too many blocks");
    lgml_launch(delta_block_prepare_kernel, dim3((unsigned)blocks), THREADS, 0, stream, qkv_c, gb, rows, records, n_blocks, C, H, G, D);
    int rc = lgml_launch_status("delta_block_prepare");
    if (rc) return rc;
    if (D <= 64) return launch_scan<16>(qkv_c, records, state, state_stride, rows, first, requests, slots, o_out, n_requests, H, G, D, Dv, stream);
    return launch_scan<32>(qkv_c, records, state, state_stride, rows, first, requests, slots, o_out, n_requests, H, G, D, Dv, stream);
}
