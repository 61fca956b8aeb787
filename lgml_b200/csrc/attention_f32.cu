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
//   * attention_f32_decode_kernel: one, two, four or eight heads of a KV head of one token a CTA (the cache is read once
//     per such run of heads), all of their keys or one chunk; a second kernel then merges the chunks.
// Which of the ways a token goes is a matter of work alone (attention_f32_short and attention_f32_chunks in ops.py).  Bound by latency at
// short contexts (a chain of copies, scores, maximum, values; no unit is half busy), by HBM at long ones in the decode kernel (32
// requests of 40 heads on 40 at 4,090 keys: 6.6 TB/s, the copy rate), and in the prompt kernel by the chains between its barriers: 11.2 us a
// block of 64 rows and keys, of which its FMAs are 4.2.
// Microseconds on one B200, heads of 128: a warp per key and a CTA per (token, head); eight heads a CTA whatever the group, branches for
// hidden keys and a lookup of the page per 16 bytes; now:
//   decode, 4 requests, 16 heads on 4, 1,030 keys 253, 27, 15; at 20 keys in a captured step (with the merge) 5.8, 9.8, 6.6;
//   decode, 32 requests, 40 on 40, 20 keys 11.5, 41, 10.5; 4,090 keys 1,665, 2,501, 813; of those a window of 256 110, 231, 61;
//   prompts of 9, 40, 300 and 1,000 tokens, 16 on 4: 4.2, 18, 5.0; 11.3, 19.7, 7.1; 191, 90, 60; 1,713, 385, 251;
//   one portion of 9 tokens beside 31 decoding requests, 40 on 40, 1,030 keys: 721, 2,412, 412.
#include <math.h>
#include <type_traits>

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
    const int *positions, *seq_of_token, *tiles, *few, *block_table;
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
__device__ __forceinline__ float finish_score(float dot, const Args &a) {
    const float v = __fmul_rn(dot, a.scale);
    return a.softcap > 0.f ? __fmul_rn(a.softcap, tanhf(__fdiv_rn(v, a.softcap))) : v;
}
__device__ __forceinline__ float finish_score(const float (&s)[4], const Args &a) {
    return finish_score(__fadd_rn(__fadd_rn(s[0], s[1]), __fadd_rn(s[2], s[3])), a);
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
// from a page that the table does not hold (flagged, and `ok` false: the key is skipped).  What is not loaded is left as it is.
template <int DP, int LD, int THREADS>
__device__ __forceinline__ void load_block(float *dst, unsigned char *ok, const float *pages, const Args &a, const int *table, int g, int kb, int first, int last) {
    constexpr int PER_ROW = DP / 4, STEP = THREADS / PER_ROW;       // (a thread stays in one column)
    const int lo = max(first - kb, 0), hi = min(last - kb, KB - 1);
    if (ok != nullptr && threadIdx.x < KB && ((int)threadIdx.x < lo || (int)threadIdx.x > hi)) ok[threadIdx.x] = 0;
    const int d = (threadIdx.x % PER_ROW) * 4;
    const bool in = d < a.D;
    if (a.page_size % KB == 0) {            // the block lies in one page
        const int blk = kb / a.page_size, page = blk < a.max_blocks ? table[blk] : -1;
        const bool have = page >= 0 && page < a.n_pages;
        if (!have && ok != nullptr && threadIdx.x == 0) atomicExch(a.status, 3);
        const float *src = have ? pages + (((size_t)page * a.Hkv + g) * a.page_size + (size_t)(kb - blk * a.page_size)) * a.D : pages;
#pragma unroll 8
        for (int r = lo + threadIdx.x / PER_ROW; r <= hi; r += STEP) {
            if (ok != nullptr && d == 0) ok[r] = have;
            cp_async_16(dst + r * LD + d, have && in ? src + (size_t)r * a.D + d : pages, have && in);
        }
        return;
    }
    for (int r = lo + threadIdx.x / PER_ROW; r <= hi; r += STEP) {
        const int j = kb + r, blk = j / a.page_size, page = blk < a.max_blocks ? table[blk] : -1;
        const bool have = page >= 0 && page < a.n_pages;
        const float *src = pages + (have ? (((size_t)page * a.Hkv + g) * a.page_size + (size_t)(j - blk * a.page_size)) * a.D : 0);
        if (ok != nullptr && d == 0) {
            if (!have) atomicExch(a.status, 3);
            ok[r] = have;
        }
        cp_async_16(dst + r * LD + d, have && in ? src + d : pages, have && in);
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
        bool all = true;                                     // do all of this thread's rows see all of its keys?
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int key = b * KB + tx + 16 * j;
                all = all && (ty * 4 + i >= n_rows || (there[j] && key >= lo[i] && key <= hi[i]));
            }
        all = __syncthreads_and(all);                        // ... and every thread has read this block's keys
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
        // (hidden keys by selection: a branch a key and row took longer than all of the additions)
        auto add_values = [&](auto checked, int k0, int k1) {
#pragma unroll 4
            for (int k = k0; k <= k1; ++k) {
                const float4 p4 = *reinterpret_cast<const float4 *>(Pr + k * LP + ty * 4);
                const float p[4] = {p4.x, p4.y, p4.z, p4.w};
                float4 v[ND];
#pragma unroll
                for (int n = 0; n < ND; ++n) v[n] = *reinterpret_cast<const float4 *>(V + k * DP + n * 64 + tx * 4);
#pragma unroll
                for (int i = 0; i < 4; ++i) {
                    const bool use = !decltype(checked)::value || !(p[i] < 0.f);
                    lb[i] = use ? __fadd_rn(lb[i], p[i]) : lb[i];
#pragma unroll
                    for (int n = 0; n < ND; ++n) {
                        float *to = o[i] + 4 * n;
                        to[0] = use ? fmaf(p[i], v[n].x, to[0]) : to[0], to[1] = use ? fmaf(p[i], v[n].y, to[1]) : to[1];
                        to[2] = use ? fmaf(p[i], v[n].z, to[2]) : to[2], to[3] = use ? fmaf(p[i], v[n].w, to[3]) : to[3];
                    }
                }
            }
        };
        if (all) add_values(std::false_type(), 0, KB - 1);
        else add_values(std::true_type(), max(first - b * KB, 0), min(last - b * KB, KB - 1));
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
constexpr int DT = 128;
template <int DP, int HP> struct Decode {
    static constexpr int LD = DP + 4;
    static constexpr size_t SMEM = sizeof(float) * (HP * LD + KB * LD + KB * DP + HP * KB + 4 * HP) + KB * 2;
};

__device__ __forceinline__ float warp_top(float v) {
    float r;
    asm("redux.sync.max.f32 %0, %1, 0xffffffff;" : "=f"(r) : "f"(v));
    return r;
}

// CTA (token, KV head and run of up to HP of its heads, and, unless WHOLE, chunk).  Scores: a thread has one key and HP / 2 heads (HP 2: one;
// HP 1: two of the four sums, its neighbour has the others).  Values: a thread has one of the head size and all heads (head size up to 64:
// half of them).
template <int DP, int HP, bool WHOLE>
__global__ void __launch_bounds__(DT) attention_f32_decode_kernel(const Args a, int n_runs, int heads_per_run, int at0) {
    using P = Decode<DP, HP>;
    constexpr int LD = P::LD, NS = HP <= 2 ? 1 : HP / 2, NV = DP == 64 && HP > 1 ? HP / 2 : HP, WARPS_OF_HEAD = HP == 1 ? 4 : 2;
    extern __shared__ __align__(16) float smem_f[];
    float *Q = smem_f, *K = Q + HP * LD, *V = K + KB * LD, *Pr = V + KB * DP, *tops = Pr + HP * KB;     // Pr [HP][KB], tops [warps of a head][HP]
    unsigned char *ok = reinterpret_cast<unsigned char *>(tops + 4 * HP);
    pdl_trigger();
    pdl_wait();
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int t = a.few ? a.few[at0 + blockIdx.x] : at0 + blockIdx.x, g = blockIdx.y / n_runs, run = blockIdx.y % n_runs;
    const int group = a.H / a.Hkv, h0 = g * group + run * heads_per_run, n_heads = min(heads_per_run, group - run * heads_per_run);
    const int pos = a.positions[t];
    const int first = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    int b0 = first / KB, b1 = pos < 0 ? -1 : pos / KB;
    if (!WHOLE) {
        const int chunk = first / CHUNK + (int)blockIdx.z;          // chunks are counted from the first that is visible
        b0 = max(b0, 2 * chunk), b1 = min(b1, 2 * chunk + 1);
        if (b0 > b1) return;                                        // (the merge does not read it)
    }
    const int *table = a.block_table + (size_t)a.seq_of_token[t] * a.max_blocks;
    if (b0 <= b1) {
        for (int c = tid; c < HP * (DP / 4); c += DT) {
            const int r = c / (DP / 4), d = (c % (DP / 4)) * 4;
            if (r < n_heads && d < a.D) cp_async_16(Q + r * LD + d, a.q + (size_t)t * a.ldq + (size_t)(h0 + r) * a.D + d, true);
        }
        load_block<DP, LD, DT>(K, ok, a.k_pages, a, table, g, b0 * KB, first, pos);
        cp_async_commit();
        load_block<DP, DP, DT>(V, nullptr, a.v_pages, a, table, g, b0 * KB, first, pos);
        cp_async_commit();
    }
    const int key = HP == 1 ? tid >> 1 : tid & 63, sh = HP == 1 ? 0 : (tid >> 6) * NS;      // scores: heads sh .. sh + NS - 1
    const int dim = tid % DP, vh = DP == 64 ? tid / 64 * NV : 0;                            // values: heads vh .. vh + NV - 1
    const bool works = dim < a.D && vh < HP;
    float ms[NS], mv[NV], l[NV], o[NV], M[NV], L[NV], O[NV];
#pragma unroll
    for (int i = 0; i < NS; ++i) ms[i] = -INFINITY;
#pragma unroll
    for (int i = 0; i < NV; ++i) mv[i] = M[i] = -INFINITY, l[i] = L[i] = o[i] = O[i] = 0.f;
    for (int b = b0; b <= b1; ++b) {
        unsigned char *okb = ok + ((b - b0) & 1) * KB, *ok_next = ok + ((b - b0 + 1) & 1) * KB;
        const int r_lo = max(first - b * KB, 0), r_hi = min(pos - b * KB, KB - 1);          // the visible rows of the block
        cp_async_wait<1>();
        __syncthreads();
        const bool seen = okb[key] != 0;
        float s[NS];
        if constexpr (HP == 1) {
            const int half = (tid & 1) * 2;
            float2 acc = make_float2(0.f, 0.f);
            if (seen) {
#pragma unroll 8
                for (int d = 0; d < a.D; d += 4) {
                    const float2 k = *reinterpret_cast<const float2 *>(K + key * LD + d + half), q = *reinterpret_cast<const float2 *>(Q + d + half);
                    acc.x = fmaf(q.x, k.x, acc.x), acc.y = fmaf(q.y, k.y, acc.y);
                }
            }
            const float part = __fadd_rn(acc.x, acc.y);
            s[0] = finish_score(__fadd_rn(part, __shfl_xor_sync(0xffffffffu, part, 1)), a);
        } else {
            float acc[NS][4];
#pragma unroll
            for (int i = 0; i < NS; ++i)
#pragma unroll
                for (int c = 0; c < 4; ++c) acc[i][c] = 0.f;
            if (seen) {
#pragma unroll 8
                for (int d = 0; d < a.D; d += 4) {
                    const float4 k = *reinterpret_cast<const float4 *>(K + key * LD + d);
#pragma unroll
                    for (int i = 0; i < NS; ++i) add_score(acc[i], *reinterpret_cast<const float4 *>(Q + (sh + i) * LD + d), k);
                }
            }
#pragma unroll
            for (int i = 0; i < NS; ++i) s[i] = finish_score(acc[i], a);
        }
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            const float top = warp_top(seen ? fmaxf(-INFINITY, s[i]) : -INFINITY);
            if (lane == 0) tops[warp % WARPS_OF_HEAD * HP + sh + i] = top;
        }
        const bool all = __syncthreads_and(seen);            // the keys are read; the warps' maxima are there
        if (b < b1) load_block<DP, LD, DT>(K, ok_next, a.k_pages, a, table, g, (b + 1) * KB, first, pos);
        cp_async_commit();
        auto new_top = [&](float m, int h) {
#pragma unroll
            for (int w = 0; w < WARPS_OF_HEAD; ++w) m = fmaxf(m, tops[w * HP + h]);
            return m;
        };
#pragma unroll
        for (int i = 0; i < NS; ++i) {
            ms[i] = new_top(ms[i], sh + i);
            const float p = prob_of(s[i], seen, ms[i]);
            if (HP > 1 || !(tid & 1)) Pr[(sh + i) * KB + key] = p;
        }
        float lb[NV];
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            lb[i] = 0.f;
            if (!works) continue;
            const float now = new_top(mv[i], vh + i), f = shrink(mv[i], now);
            mv[i] = now, l[i] = __fmul_rn(l[i], f), o[i] = __fmul_rn(o[i], f);
        }
        cp_async_wait<1>();
        __syncthreads();                                     // values and probabilities are there; the maxima are read
        auto add_values = [&](auto checked, int k0, int k1) {
#pragma unroll 4
            for (int k = k0; k <= k1; k += 4) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) v[u] = V[(k + u) * DP + dim];
#pragma unroll
                for (int i = 0; i < NV; ++i) {
                    const float4 p4 = *reinterpret_cast<const float4 *>(Pr + (vh + i) * KB + k);
                    const float p[4] = {p4.x, p4.y, p4.z, p4.w};
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const bool use = !decltype(checked)::value || !(p[u] < 0.f);
                        lb[i] = use ? __fadd_rn(lb[i], p[u]) : lb[i];
                        o[i] = use ? fmaf(p[u], v[u], o[i]) : o[i];
                    }
                }
            }
        };
        if (works) {
            if (all) add_values(std::false_type(), 0, KB - 1);
            else add_values(std::true_type(), r_lo & ~3, r_hi);
        }
        __syncthreads();
        if (b < b1) load_block<DP, DP, DT>(V, nullptr, a.v_pages, a, table, g, (b + 1) * KB, first, pos);
        cp_async_commit();
        const bool ends = (b & 1) || b == b1;                // the chunk's second block, or the last there is
#pragma unroll
        for (int i = 0; i < NV; ++i) {
            l[i] = __fadd_rn(l[i], lb[i]);
            float f_old, f_new;
            if (!WHOLE || !ends) continue;
            if (merge_ml(M[i], L[i], mv[i], l[i], f_old, f_new)) O[i] = merge_o(O[i], o[i], f_old, f_new);
            mv[i] = -INFINITY, l[i] = o[i] = 0.f;
        }
        if (WHOLE && ends) {
#pragma unroll
            for (int i = 0; i < NS; ++i) ms[i] = -INFINITY;
        }
    }
    cp_async_wait<0>();
    if (!works) return;
#pragma unroll
    for (int i = 0; i < NV; ++i) {
        const int h = vh + i;
        if (h >= n_heads) continue;
        if (WHOLE) {
            a.out[(size_t)t * a.ldo + (size_t)(h0 + h) * a.D + dim] = finish_out(O[i], L[i]);
        } else {
            const size_t at = ((size_t)blockIdx.x * a.H + h0 + h) * a.n_chunks + blockIdx.z;
            a.part_o[at * a.D + dim] = o[i];
            if (dim == 0) a.part_ml[at] = make_float2(mv[i], l[i]);
        }
    }
}

// One warp per (token, head): its chunks in order, four of the head size a lane.
__global__ void __launch_bounds__(128) attention_f32_merge_kernel(const Args a, int n_tokens, int at0) {
    pdl_trigger();
    pdl_wait();
    const int u = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (u >= n_tokens * a.H) return;
    const int at_token = u / a.H, h = u - at_token * a.H, t = a.few ? a.few[at0 + at_token] : at0 + at_token;
    const int pos = a.positions[t];
    const int first = (a.window > 0 && pos - a.window + 1 > 0) ? pos - a.window + 1 : 0;
    const int n = pos < 0 ? 0 : min(pos / CHUNK - first / CHUNK + 1, a.n_chunks);
    const int d = lane * 4;
    float M = -INFINITY, L = 0.f, O[4] = {0.f, 0.f, 0.f, 0.f};
    for (int c = 0; c < n; c += 4) {
        float2 ml[4];
        float4 o[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const size_t at = (size_t)u * a.n_chunks + min(c + i, n - 1);
            ml[i] = act_load(reinterpret_cast<const float2 *>(a.part_ml + at));
            o[i] = d < a.D ? act_load(reinterpret_cast<const float4 *>(a.part_o + at * a.D + d)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            float f_old, f_new;
            if (c + i < n && merge_ml(M, L, ml[i].x, ml[i].y, f_old, f_new)) {
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

// n tokens, `per` at a time where the scratch holds no more (the next ones wait for the merge of those ahead).
template <int DP, int HP, bool WHOLE> int run_decode(const Args &a, int n, int per, cudaStream_t stream) {
    auto kernel = attention_f32_decode_kernel<DP, HP, WHOLE>;
    if (allow_smem(kernel, Decode<DP, HP>::SMEM)) return -1;
    const int group = a.H / a.Hkv, runs = (group + 7) / 8, heads = (group + runs - 1) / runs;
    for (int at = 0; at < n; at += per) {
        const int m = min(per, n - at);
        lgml_launch(kernel, dim3(m, a.Hkv * runs, WHOLE ? 1 : a.n_chunks), DT, Decode<DP, HP>::SMEM, stream, a, runs, heads, at);
        int rc = lgml_launch_status("attention_f32 decode");
        if (rc || WHOLE) {
            if (rc) return rc;
            continue;
        }
        lgml_launch(attention_f32_merge_kernel, dim3(((long long)m * a.H + 3) / 4), 128, 0, stream, a, m, at);
        if ((rc = lgml_launch_status("attention_f32 merge"))) return rc;
    }
    return 0;
}
template <int DP, bool WHOLE> int run_decode_heads(const Args &a, int n, int per, cudaStream_t stream) {
    const int group = a.H / a.Hkv, runs = (group + 7) / 8, heads = (group + runs - 1) / runs;
    if (heads == 1) return run_decode<DP, 1, WHOLE>(a, n, per, stream);
    if (heads == 2) return run_decode<DP, 2, WHOLE>(a, n, per, stream);
    return heads <= 4 ? run_decode<DP, 4, WHOLE>(a, n, per, stream) : run_decode<DP, 8, WHOLE>(a, n, per, stream);
}
}  // namespace

LGML_API int lgml_attention_f32_chunk(void) { return CHUNK; }

// `tiles` (n_tiles of them), int32 [n_tiles, 4] rows (request row, first token row, tokens, 0): tokens of prompts and portions, a tile within
// one request, at most 64 / (H / Hkv) tokens.  `few` (n_few; null: rows 0 .. n_few - 1): rows of tokens that are taken each by itself.
// n_chunks 0: such a token's keys one after the other; else side by side in n_chunks chunks (as many as the longest context or window
// touches), with scratch for scratch_tokens tokens: part_o and part_ml hold scratch_tokens * H * n_chunks rows of D floats and of two.
LGML_API int lgml_attention_f32(const float *q, int ldq, const int *positions, const int *seq_of_token, const int *tiles, int n_tiles, const int *few, int n_few,
                                const int *block_table, int max_blocks, const float *k_pages, const float *v_pages, int n_pages, int page_size,
                                float *out, int ldo, int H, int Hkv, int D, float scale, int window, float softcap, int n_chunks, int scratch_tokens,
                                float *part_o, float *part_ml, int *status, cudaStream_t stream) {
    LGML_REQUIRE(n_tiles >= 0 && n_few >= 0 && H > 0 && Hkv > 0 && D > 0 && page_size > 0 && max_blocks > 0, "attention_f32: bad sizes");
    LGML_REQUIRE(H % Hkv == 0 && H / Hkv <= ROWS, "attention_f32: %d heads on %d KV heads", H, Hkv);
    LGML_REQUIRE(D % 4 == 0 && D <= 128, "attention_f32: head_dim %d is no multiple of 4 up to 128", D);
    LGML_REQUIRE(ldq % 4 == 0 && ldo % 4 == 0 && (((uintptr_t)q | (uintptr_t)out | (uintptr_t)k_pages | (uintptr_t)v_pages) & 15) == 0,
                 "attention_f32: rows must start on 16 bytes");
    LGML_REQUIRE(window >= 0 && softcap >= 0.f && n_chunks >= 0, "attention_f32: bad window, cap or chunks");
    LGML_REQUIRE(n_chunks <= 65535 && (long long)Hkv * ((H / Hkv + 7) / 8) <= 65535, "attention_f32: grid too large");
    LGML_REQUIRE(n_chunks == 0 || (scratch_tokens > 0 && part_o != nullptr && part_ml != nullptr && (((uintptr_t)part_o | (uintptr_t)part_ml) & 15) == 0),
                 "attention_f32: several chunks need scratch memory");
    const Args a = {q, ldq, positions, seq_of_token, tiles, few, block_table, max_blocks, k_pages, v_pages, n_pages, page_size, out, ldo,
                    part_o, (float2 *)part_ml, n_chunks, H, Hkv, D, scale, window, softcap, status};
    if (n_tiles > 0) {
        const int rc = D <= 64 ? run_prompt<64>(a, n_tiles, stream) : run_prompt<128>(a, n_tiles, stream);
        if (rc) return rc;
    }
    if (n_few == 0) return 0;
    if (n_chunks == 0) return D <= 64 ? run_decode_heads<64, true>(a, n_few, n_few, stream) : run_decode_heads<128, true>(a, n_few, n_few, stream);
    return D <= 64 ? run_decode_heads<64, false>(a, n_few, scratch_tokens, stream) : run_decode_heads<128, false>(a, n_few, scratch_tokens, stream);
}
