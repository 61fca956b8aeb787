// Paged attention of the 32-bit path: float32 queries, keys, values, scores and sums, no tensor cores.
// softmax over keys of (q . k) * scale with keys at positions <= the query's, an optional window and
// score cap (lua/lgml/transformer.lua:1805-1816, src/lgml.c:2083-2118; head h reads KV head h / (H / Hkv)).
//
// A (token, head)'s result has the same bits however its request was cut into steps and whatever else is
// in the batch.  Both kernels below therefore do one arithmetic, told by absolute positions:
//   * a score is four sums over d = c, c + 4, c + 8, ... (c = 0 .. 3) added as (0 + 1) + (2 + 3);
//   * keys come in blocks of 64 (positions 64 b ..), a running maximum from block to block; inside a
//     block probabilities and weighted values are added key by key;
//   * two blocks are a chunk with a maximum, sum and values of its own, and the chunks are merged one
//     after the other, the earliest first.
// What is between them is only who does it:
//   * attention_f32_prompt_kernel: 64 rows (tokens x heads of one KV head) a CTA, all of their keys: every
//     key and value is read from shared memory for 64 rows.  Scores 4 x 4 a thread, values 4 x 8.
//   * attention_f32_decode_kernel: up to eight heads of one token and one chunk a CTA, so that few tokens
//     fill the chip; a second kernel merges the chunks.  The cache is read once for the heads that share it.
// Before, a warp per key and a CTA per (token, head): no key was ever shared, and 4 requests of 16 heads
// ran on 64 CTAs whatever their context.  Measured on one B200 in two layers of 16 heads of 128 on 4: a decode step of
// 4 requests at 1,030 keys 1.0 -> 0.38 ms (attention 0.33 -> 0.02 ms a layer), prompts of 300 and 600 tokens 9.5 -> 7.2 ms.
#include <math.h>

#include "common.cuh"

LGML_DEFINE_LAST_ERROR(lgml_attention_f32)

namespace {
constexpr int KB = 64;               // keys of a block
constexpr int CHUNK = 2 * KB;        // keys of a chunk

__device__ __forceinline__ void cp_async_16(float *dst, const float *src, bool valid) {
    const int bytes = valid ? 16 : 0;   // 0: the 16 bytes are filled with zeros
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src), "r"(bytes) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

struct Args {
    const float *q;
    int ldq;
    const int *positions, *seq_of_token, *tiles, *block_table;
    int max_blocks;
    const float *k_pages, *v_pages;
    int n_pages, page_size;
    float *out;
    int ldo;
    float *part_o;          // [tokens, H, n_chunks, D]
    float2 *part_ml;        // [tokens, H, n_chunks]: maximum, sum
    int n_chunks, H, Hkv, D;
    float scale;
    int window;
    float softcap;
    int *status;
};

// ---- the shared arithmetic; every rounding is written out, so that no kernel's compiler contracts another pair ----
__device__ __forceinline__ float finish_score(const float (&s)[4], const Args &a) {
    const float dot = __fadd_rn(__fadd_rn(s[0], s[1]), __fadd_rn(s[2], s[3]));
    const float v = __fmul_rn(dot, a.scale);
    return a.softcap > 0.f ? __fmul_rn(a.softcap, tanhf(__fdiv_rn(v, a.softcap))) : v;
}
__device__ __forceinline__ void add_score(float (&s)[4], float4 q, float4 k) {
    s[0] = fmaf(q.x, k.x, s[0]), s[1] = fmaf(q.y, k.y, s[1]), s[2] = fmaf(q.z, k.z, s[2]), s[3] = fmaf(q.w, k.w, s[3]);
}
// A key's probability; hidden keys are marked -1 (their values are not touched, whatever they hold).  While every score of the
// chunk so far is -inf so is the maximum, and -inf less -inf is no number: such a key's probability is 0, and the chunk is merged
// as one without visible keys.
__device__ __forceinline__ float prob_of(float s, bool seen, float m) { return seen ? expf(__fsub_rn(s, m == -INFINITY ? 0.f : m)) : -1.f; }
__device__ __forceinline__ float shrink(float m_old, float m_new) { return m_old == m_new ? 1.f : expf(__fsub_rn(m_old, m_new)); }
// merge a chunk's (m, l) into the running (M, L): the factors of what was there and of what comes
__device__ __forceinline__ bool merge_ml(float &M, float &L, float m, float l, float &f_old, float &f_new) {
    if (m == -INFINITY && l == 0.f) return false;       // no key of the chunk was visible
    const float top = fmaxf(M, m);
    f_old = M == -INFINITY ? 0.f : expf(__fsub_rn(M, top));
    f_new = m == top ? 1.f : expf(__fsub_rn(m, top));
    L = __fadd_rn(__fmul_rn(L, f_old), __fmul_rn(l, f_new));
    M = top;
    return true;
}
__device__ __forceinline__ float merge_o(float O, float o, float f_old, float f_new) { return __fadd_rn(__fmul_rn(O, f_old), __fmul_rn(o, f_new)); }
__device__ __forceinline__ float finish_out(float O, float L) { return L > 0.f ? __fdiv_rn(O, L) : 0.f; }

// Rows `kb` .. of keys or values into shared memory, LD floats apart; nothing past `last`, below `first` or
// from a page that the table does not hold (flagged, and `ok` false: the key is skipped).
template <int DP, int LD, int THREADS>
__device__ __forceinline__ void load_block(float *dst, unsigned char *ok, const float *pages, const Args &a, const int *table, int g, int kb, int first, int last) {
    constexpr int PER_ROW = DP / 4;
#pragma unroll 4
    for (int c = threadIdx.x; c < KB * PER_ROW; c += THREADS) {
        const int r = c / PER_ROW, d = (c % PER_ROW) * 4;
        const int j = kb + r;
        const float *src = pages;
        bool have = false;
        if (j >= first && j <= last) {
            const int blk = j / a.page_size;
            const int page = blk < a.max_blocks ? table[blk] : -1;
            have = page >= 0 && page < a.n_pages;
            if (have) src += (((size_t)page * a.Hkv + g) * a.page_size + (size_t)(j - blk * a.page_size)) * a.D;
            else if (ok != nullptr && d == 0) atomicExch(a.status, 3);
        }
        if (ok != nullptr && d == 0) ok[r] = have;
        const bool in = have && d < a.D;
        cp_async_16(dst + r * LD + d, in ? src + d : pages, in);
    }
}

// ---- prompts -------------------------------------------------------------------------------------
constexpr int PT = 256, ROWS = 64;
template <int DP> struct Prompt {
    static constexpr int LD = DP + 4, LP = ROWS + 4;
    static constexpr size_t SMEM = sizeof(float) * (ROWS * LD + KB * LD + KB * DP + KB * LP) + KB * 2;
};

template <int DP> __global__ void __launch_bounds__(PT) attention_f32_prompt_kernel(const Args a) {
    using P = Prompt<DP>;
    constexpr int LD = P::LD, LP = P::LP, ND = DP / 64;      // ND groups of four values a thread
    extern __shared__ __align__(16) float smem_f[];
    float *Q = smem_f, *K = Q + ROWS * LD, *V = K + KB * LD, *Pr = V + KB * DP;
    unsigned char *ok = reinterpret_cast<unsigned char *>(Pr + KB * LP);        // two blocks' flags: K of the next is copied early
    pdl_wait();
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int seq = a.tiles[4 * blockIdx.x], t0 = a.tiles[4 * blockIdx.x + 1], nt = a.tiles[4 * blockIdx.x + 2];
    const int g = blockIdx.y, group = a.H / a.Hkv;
    const int n_rows = nt * group;                           // row = token * group + head of the group
    const int *table = a.block_table + (size_t)seq * a.max_blocks;
    const int pos0 = a.positions[t0], last = a.positions[t0 + nt - 1];
    const int first = (a.window > 0 && pos0 - a.window + 1 > 0) ? pos0 - a.window + 1 : 0;
    const int b0 = first / KB, b1 = last / KB;
    for (int c = tid; c < ROWS * (DP / 4); c += PT) {
        const int r = c / (DP / 4), d = (c % (DP / 4)) * 4;
        const bool in = r < n_rows && d < a.D;
        cp_async_16(Q + r * LD + d, in ? a.q + (size_t)(t0 + r / group) * a.ldq + (size_t)(g * group + r % group) * a.D + d : a.q, in);
    }
    load_block<DP, LD, PT>(K, ok, a.k_pages, a, table, g, b0 * KB, first, last);
    cp_async_commit();
    load_block<DP, DP, PT>(V, nullptr, a.v_pages, a, table, g, b0 * KB, first, last);
    cp_async_commit();

    int lo[4], hi[4];                                        // the keys each of this thread's rows sees
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        hi[i] = r < n_rows ? a.positions[t0 + r / group] : -1;
        lo[i] = (a.window > 0 && hi[i] - a.window + 1 > 0) ? hi[i] - a.window + 1 : 0;
    }
    float m[4], l[4], M[4], L[4], o[4][4 * ND], O[4][4 * ND];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        m[i] = M[i] = -INFINITY, l[i] = L[i] = 0.f;
#pragma unroll
        for (int d = 0; d < 4 * ND; ++d) o[i][d] = O[i][d] = 0.f;
    }
    for (int b = b0; b <= b1; ++b) {
        unsigned char *okb = ok + ((b - b0) & 1) * KB, *ok_next = ok + ((b - b0 + 1) & 1) * KB;
        cp_async_wait<1>();                                  // keys are there (values may be under way)
        __syncthreads();
        float s[4][4];
        {
            float acc[4][4][4];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int c = 0; c < 4; ++c) acc[i][j][c] = 0.f;
#pragma unroll 4
            for (int d = 0; d < DP; d += 4) {
                float4 k[4];
#pragma unroll
                for (int j = 0; j < 4; ++j) k[j] = *reinterpret_cast<const float4 *>(K + (tx + 16 * j) * LD + d);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const float4 q = *reinterpret_cast<const float4 *>(Q + (ty * 4 + i) * LD + d);
#pragma unroll
                    for (int j = 0; j < 4; ++j) add_score(acc[i][j], q, k[j]);
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) s[i][j] = finish_score(acc[i][j], a);
        }
        bool there[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) there[j] = okb[tx + 16 * j] != 0;
        __syncthreads();                                     // every thread has read this block's keys
        if (b < b1) load_block<DP, LD, PT>(K, ok_next, a.k_pages, a, table, g, (b + 1) * KB, first, last);
        cp_async_commit();
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float top = -INFINITY;
            bool seen[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = b * KB + tx + 16 * j;
                seen[j] = there[j] && key >= lo[i] && key <= hi[i];
                if (seen[j]) top = fmaxf(top, s[i][j]);
            }
#pragma unroll
            for (int x = 1; x < 16; x <<= 1) top = fmaxf(top, __shfl_xor_sync(0xffffffffu, top, x));
            const float now = fmaxf(m[i], top);
#pragma unroll
            for (int j = 0; j < 4; ++j) s[i][j] = prob_of(s[i][j], seen[j], now);
            const float f = shrink(m[i], now);
            m[i] = now;
            l[i] = __fmul_rn(l[i], f);
#pragma unroll
            for (int d = 0; d < 4 * ND; ++d) o[i][d] = __fmul_rn(o[i][d], f);
        }
        // the sixteen lanes of a row write and read the row's probabilities among themselves
#pragma unroll
        for (int j = 0; j < 4; ++j) *reinterpret_cast<float4 *>(Pr + (tx + 16 * j) * LP + ty * 4) = make_float4(s[0][j], s[1][j], s[2][j], s[3][j]);
        cp_async_wait<1>();                                  // values are there
        __syncthreads();
        float lb[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
        for (int k = 0; k < KB; ++k) {
            const float4 p4 = *reinterpret_cast<const float4 *>(Pr + k * LP + ty * 4);
            const float p[4] = {p4.x, p4.y, p4.z, p4.w};
            float4 v[ND];
#pragma unroll
            for (int n = 0; n < ND; ++n) v[n] = *reinterpret_cast<const float4 *>(V + k * DP + n * 64 + tx * 4);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if (!(p[i] < 0.f)) {
                    lb[i] = __fadd_rn(lb[i], p[i]);
#pragma unroll
                    for (int n = 0; n < ND; ++n) {
                        o[i][4 * n] = fmaf(p[i], v[n].x, o[i][4 * n]), o[i][4 * n + 1] = fmaf(p[i], v[n].y, o[i][4 * n + 1]);
                        o[i][4 * n + 2] = fmaf(p[i], v[n].z, o[i][4 * n + 2]), o[i][4 * n + 3] = fmaf(p[i], v[n].w, o[i][4 * n + 3]);
                    }
                }
            }
        }
        __syncthreads();                                     // every thread has read this block's values
        if (b < b1) load_block<DP, DP, PT>(V, nullptr, a.v_pages, a, table, g, (b + 1) * KB, first, last);
        cp_async_commit();
        const bool ends = (b & 1) || b == b1;                // the chunk's second block, or the last there is
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            l[i] = __fadd_rn(l[i], lb[i]);
            if (ends) {
                float f_old, f_new;
                if (merge_ml(M[i], L[i], m[i], l[i], f_old, f_new)) {
#pragma unroll
                    for (int d = 0; d < 4 * ND; ++d) O[i][d] = merge_o(O[i][d], o[i][d], f_old, f_new);
                }
                m[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
                for (int d = 0; d < 4 * ND; ++d) o[i][d] = 0.f;
            }
        }
    }
    cp_async_wait<0>();
    pdl_trigger();      // at the end: a CTA takes half of an SM's shared memory and more
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const int r = ty * 4 + i;
        if (r >= n_rows) continue;
        float *dst = a.out + (size_t)(t0 + r / group) * a.ldo + (size_t)(g * group + r % group) * a.D;
#pragma unroll
        for (int n = 0; n < ND; ++n) {
            const int d = n * 64 + tx * 4;
            if (d < a.D)
                *reinterpret_cast<float4 *>(dst + d) = make_float4(finish_out(O[i][4 * n], L[i]), finish_out(O[i][4 * n + 1], L[i]),
                                                                   finish_out(O[i][4 * n + 2], L[i]), finish_out(O[i][4 * n + 3], L[i]));
        }
    }
}

// ---- few tokens ----------------------------------------------------------------------------------
constexpr int DT = 128, HEADS = 8;
template <int DP> struct Decode {
    static constexpr int LD = DP + 4, LP = HEADS + 4;
    static constexpr size_t SMEM = sizeof(float) * (HEADS * LD + KB * LD + KB * DP + KB * LP + 8 * 2) + KB * 2;
};

// CTA (token, KV head and run of eight of its heads, chunk).  Scores: thread = key tid % 64, four heads.  Values:
// thread = four of the head size and DP / 64 heads (DP 128: lane and two heads a warp; DP 64: half a warp and one head).
template <int DP> __global__ void __launch_bounds__(DT) attention_f32_decode_kernel(const Args a, int head_runs) {
    using P = Decode<DP>;
    constexpr int LD = P::LD, LP = P::LP, NH = DP / 64;
    extern __shared__ __align__(16) float smem_f[];
    float *Q = smem_f, *K = Q + HEADS * LD, *V = K + KB * LD, *Pr = V + KB * DP, *tops = Pr + KB * LP;      // tops [2 warps of a head][8]
    unsigned char *ok = reinterpret_cast<unsigned char *>(tops + 16);
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = blockIdx.x, g = blockIdx.y / head_runs, run = blockIdx.y % head_runs, chunk = blockIdx.z;
    const int group = a.H / a.Hkv, h0 = g * group + run * HEADS, n_heads = min(HEADS, group - run * HEADS);
    const int pos = a.positions[t];
    const int first = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int b0 = max(chunk * 2, first / KB), b1 = min(chunk * 2 + 1, pos / KB);
    if (b0 > b1) {                              // no key of this chunk is visible
        if (tid < n_heads && a.n_chunks > 1) a.part_ml[((size_t)t * a.H + h0 + tid) * a.n_chunks + chunk] = make_float2(-INFINITY, 0.f);
        return;
    }
    const int *table = a.block_table + (size_t)a.seq_of_token[t] * a.max_blocks;
    for (int c = tid; c < HEADS * (DP / 4); c += DT) {
        const int r = c / (DP / 4), d = (c % (DP / 4)) * 4;
        const bool in = r < n_heads && d < a.D;
        cp_async_16(Q + r * LD + d, in ? a.q + (size_t)t * a.ldq + (size_t)(h0 + r) * a.D + d : a.q, in);
    }
    load_block<DP, LD, DT>(K, ok, a.k_pages, a, table, g, b0 * KB, first, pos);
    cp_async_commit();
    load_block<DP, DP, DT>(V, nullptr, a.v_pages, a, table, g, b0 * KB, first, pos);
    cp_async_commit();
    const int key = tid & 63, sh = (tid >> 6) * 4;                  // scores: heads sh .. sh + 3
    const int d4 = (tid % (DP / 4)) * 4, vh = tid / (DP / 4) * NH;  // values: heads vh .. vh + NH - 1
    float ms[4], mv[NH], l[NH], o[NH][4];
#pragma unroll
    for (int i = 0; i < 4; ++i) ms[i] = -INFINITY;
#pragma unroll
    for (int i = 0; i < NH; ++i) {
        mv[i] = -INFINITY, l[i] = 0.f;
#pragma unroll
        for (int d = 0; d < 4; ++d) o[i][d] = 0.f;
    }
    for (int b = b0; b <= b1; ++b) {
        unsigned char *okb = ok + (b - b0) * KB;
        cp_async_wait<1>();
        __syncthreads();
        float acc[4][4];
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
#pragma unroll 8
        for (int d = 0; d < DP; d += 4) {
            const float4 k = *reinterpret_cast<const float4 *>(K + key * LD + d);
#pragma unroll
            for (int i = 0; i < 4; ++i) add_score(acc[i], *reinterpret_cast<const float4 *>(Q + (sh + i) * LD + d), k);
        }
        const int j = b * KB + key;
        const bool seen = okb[key] != 0 && j >= first && j <= pos;
        float s[4], top[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            s[i] = finish_score(acc[i], a);
            top[i] = seen ? fmaxf(-INFINITY, s[i]) : -INFINITY;
#pragma unroll
            for (int x = 16; x > 0; x >>= 1) top[i] = fmaxf(top[i], __shfl_xor_sync(0xffffffffu, top[i], x));
            if (lane == 0) tops[(warp & 1) * 8 + sh + i] = top[i];
        }
        __syncthreads();                                     // the keys are read; both warps' maxima are there
        if (b < b1) load_block<DP, LD, DT>(K, okb + KB, a.k_pages, a, table, g, (b + 1) * KB, first, pos);
        cp_async_commit();
        float pr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            ms[i] = fmaxf(ms[i], fmaxf(tops[sh + i], tops[8 + sh + i]));
            pr[i] = prob_of(s[i], seen, ms[i]);
        }
        *reinterpret_cast<float4 *>(Pr + key * LP + sh) = make_float4(pr[0], pr[1], pr[2], pr[3]);
        float lb[NH];
#pragma unroll
        for (int i = 0; i < NH; ++i) {
            const float now = fmaxf(mv[i], fmaxf(tops[vh + i], tops[8 + vh + i])), f = shrink(mv[i], now);
            mv[i] = now, lb[i] = 0.f;
            l[i] = __fmul_rn(l[i], f);
#pragma unroll
            for (int d = 0; d < 4; ++d) o[i][d] = __fmul_rn(o[i][d], f);
        }
        cp_async_wait<1>();
        __syncthreads();                                     // values and probabilities are there; the maxima are read
#pragma unroll 8
        for (int k = 0; k < KB; ++k) {
            const float4 v = *reinterpret_cast<const float4 *>(V + k * DP + d4);
#pragma unroll
            for (int i = 0; i < NH; ++i) {
                const float p = Pr[k * LP + vh + i];
                if (!(p < 0.f)) {
                    lb[i] = __fadd_rn(lb[i], p);
                    o[i][0] = fmaf(p, v.x, o[i][0]), o[i][1] = fmaf(p, v.y, o[i][1]), o[i][2] = fmaf(p, v.z, o[i][2]), o[i][3] = fmaf(p, v.w, o[i][3]);
                }
            }
        }
        __syncthreads();
        if (b < b1) load_block<DP, DP, DT>(V, nullptr, a.v_pages, a, table, g, (b + 1) * KB, first, pos);
        cp_async_commit();
#pragma unroll
        for (int i = 0; i < NH; ++i) l[i] = __fadd_rn(l[i], lb[i]);
    }
    cp_async_wait<0>();
#pragma unroll
    for (int i = 0; i < NH; ++i) {
        const int h = vh + i;
        if (h >= n_heads || d4 >= a.D) continue;
        if (a.n_chunks == 1) {
            float M = -INFINITY, L = 0.f, f_old = 0.f, f_new = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
            if (merge_ml(M, L, mv[i], l[i], f_old, f_new)) {
#pragma unroll
                for (int d = 0; d < 4; ++d) O[d] = merge_o(0.f, o[i][d], f_old, f_new);
            }
            *reinterpret_cast<float4 *>(a.out + (size_t)t * a.ldo + (size_t)(h0 + h) * a.D + d4) =
                make_float4(finish_out(O[0], L), finish_out(O[1], L), finish_out(O[2], L), finish_out(O[3], L));
        } else {
            const size_t at = ((size_t)t * a.H + h0 + h) * a.n_chunks + chunk;
            *reinterpret_cast<float4 *>(a.part_o + at * a.D + d4) = make_float4(o[i][0], o[i][1], o[i][2], o[i][3]);
            if (d4 == 0) a.part_ml[at] = make_float2(mv[i], l[i]);
        }
    }
}

// One warp per (token, head): its chunks in order, four of the head size a lane.
__global__ void __launch_bounds__(128) attention_f32_merge_kernel(const Args a, int n_tokens) {
    pdl_trigger();
    pdl_wait();
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (u >= n_tokens * a.H) return;
    const int t = u / a.H, h = u - t * a.H;
    const int pos = a.positions[t];
    const int first = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int c0 = first / CHUNK, c1 = min(pos / CHUNK, a.n_chunks - 1);
    const int d = lane * 4;
    float M = -INFINITY, L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = c0; c <= c1; c += 4) {
        float2 ml[4];
        float4 o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const size_t at = (size_t)u * a.n_chunks + min(c + i, c1);
            ml[i] = act_load(reinterpret_cast<const float2 *>(a.part_ml + at));
            o[i] = d < a.D && (ml[i].x != -INFINITY || ml[i].y != 0.f) ? act_load(reinterpret_cast<const float4 *>(a.part_o + at * a.D + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float f_old, f_new;
            if (c + i <= c1 && merge_ml(M, L, ml[i].x, ml[i].y, f_old, f_new)) {
                O[0] = merge_o(O[0], o[i].x, f_old, f_new), O[1] = merge_o(O[1], o[i].y, f_old, f_new);
                O[2] = merge_o(O[2], o[i].z, f_old, f_new), O[3] = merge_o(O[3], o[i].w, f_old, f_new);
            }
        }
    }
    if (d < a.D)
        *reinterpret_cast<float4 *>(a.out + (size_t)t * a.ldo + (size_t)h * a.D + d) = make_float4(finish_out(O[0], L), finish_out(O[1], L), finish_out(O[2], L), finish_out(O[3], L));
}

// (At every launch: the attribute belongs to the kernel on the current device, and a process may use several.)
template <typename Kernel> int allow_smem(Kernel kernel, size_t smem) {
    if (smem <= 48 * 1024) return 0;
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) LGML_FAIL("attention_f32: cannot have %zu bytes of shared memory: %s", smem, cudaGetErrorString(e));
    return 0;
}

template <int DP> int run_prompt(const Args &a, int n_tiles, cudaStream_t stream) {
    if (allow_smem(attention_f32_prompt_kernel<DP>, Prompt<DP>::SMEM)) return -1;
    lgml_launch_alone(attention_f32_prompt_kernel<DP>, dim3(n_tiles, a.Hkv), PT, Prompt<DP>::SMEM, stream, a);
    return lgml_launch_status("attention_f32 prompt");
}

template <int DP> int run_decode(const Args &a, int n_tokens, cudaStream_t stream) {
    if (allow_smem(attention_f32_decode_kernel<DP>, Decode<DP>::SMEM)) return -1;
    const int runs = (a.H / a.Hkv + HEADS - 1) / HEADS;
    // (alone: behind the kernel that writes the cells its CTAs came to lie two and three an SM, 28.5 us instead of 22.8)
    lgml_launch_alone(attention_f32_decode_kernel<DP>, dim3(n_tokens, a.Hkv * runs, a.n_chunks), DT, Decode<DP>::SMEM, stream, a, runs);
    int rc = lgml_launch_status("attention_f32 decode");
    if (rc || a.n_chunks == 1) return rc;
    lgml_launch(attention_f32_merge_kernel, dim3((n_tokens * a.H + 3) / 4), 128, 0, stream, a, n_tokens);
    return lgml_launch_status("attention_f32 merge");
}
}  // namespace

LGML_API int lgml_attention_f32_chunk(void) { return CHUNK; }

// `tiles` (n_tiles > 0): prompts and portions, int32 [n_tiles, 4] rows (request row, first token row, tokens, 0), a tile
// within one request, at most 64 / (H / Hkv) tokens.  n_tiles = 0: every token by itself, its keys in n_chunks chunks
// (as many as the longest context has); part_o and part_ml hold n_tokens * H * n_chunks rows of D floats and of two.
LGML_API int lgml_attention_f32(const float *q, int ldq, const int *positions, const int *seq_of_token, const int *tiles, int n_tiles,
                                const int *block_table, int max_blocks, const float *k_pages, const float *v_pages, int n_pages, int page_size,
                                float *out, int ldo, int n_tokens, int H, int Hkv, int D, float scale, int window, float softcap, int n_chunks,
                                float *part_o, float *part_ml, int *status, cudaStream_t stream) {
    LGML_REQUIRE(n_tokens >= 0 && H > 0 && Hkv > 0 && D > 0 && page_size > 0 && max_blocks > 0, "attention_f32: bad sizes");
    LGML_REQUIRE(H % Hkv == 0 && H / Hkv <= ROWS, "attention_f32: %d heads on %d KV heads", H, Hkv);
    LGML_REQUIRE(D % 4 == 0 && D <= 128, "attention_f32: head_dim %d is no multiple of 4 up to 128", D);
    LGML_REQUIRE(ldq % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0,
                 "attention_f32: rows must start on 16 bytes");
    LGML_REQUIRE(window >= 0 && softcap >= 0.f && n_chunks >= 1 && n_tiles >= 0, "attention_f32: bad window, cap or chunks");
    LGML_REQUIRE(n_chunks <= 65535 && (long long)Hkv * ((H / Hkv + HEADS - 1) / HEADS) <= 65535, "attention_f32: grid too large");
    LGML_REQUIRE(n_tiles > 0 || n_chunks == 1 || (part_o != nullptr && part_ml != nullptr && (((uintptr_t)part_o | (uintptr_t)part_ml) & 15) == 0),
                 "attention_f32: several chunks need scratch memory");
    if (n_tokens == 0) return 0;
    const Args a = {q, ldq, positions, seq_of_token, tiles, block_table, max_blocks, k_pages, v_pages, n_pages, page_size, out, ldo,
                    part_o, (float2 *)part_ml, n_chunks, H, Hkv, D, scale, window, softcap, status};
    if (n_tiles > 0) return D <= 64 ? run_prompt<64>(a, n_tiles, stream) : run_prompt<128>(a, n_tiles, stream);
    return D <= 64 ? run_decode<64>(a, n_tokens, stream) : run_decode<128>(a, n_tokens, stream);
}
