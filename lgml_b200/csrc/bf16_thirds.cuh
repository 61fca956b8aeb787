// float32 products on the tensor cores, both operands in three bfloat16 parts: x = h + m + l exactly, h being the first 8 of x's 24 bits, m the
// next 8 and l the last (below 2^-110 a part is cut at 2^-133, the last bit of the smallest bfloat16 number).  Of the nine products of two
// such sums only l l is left out, under 2^-30 of a product.  A run of 16 k is two sums by mma.sync (m16n8k16) from zero, the small products
// (l m, m l, l h, h l, m m, m h, h m; under 2^-5 of the whole) and h h, that join the caller's float32 sum one after the other.  The tensor core cuts what
// it adds instead of rounding it: so little is added up there that this shows in the last place of a run at most, and a product
// that stands alone in its run is rounded once, as by an FMA (h h has 16 bits).
#pragma once
#include <stdint.h>

// two float32 operations an instruction (a product holds the scheduler for its eight cycles, so what is issued beside it counts in full)
__device__ __forceinline__ float2 add_two(float2 a, float2 b) {
    float2 r;
    asm("{.reg .b64 a, b; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; add.rn.f32x2 a, a, b; mov.b64 {%0, %1}, a;}" : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y));
    return r;
}
// a - b, where that is exact
__device__ __forceinline__ float2 less_two(float2 a, float2 b) {
    float2 r;
    asm("{.reg .b64 a, b, c; mov.b64 a, {%2, %3}; mov.b64 b, {%4, %5}; mov.b64 c, {%6, %6}; fma.rn.f32x2 a, b, c, a; mov.b64 {%0, %1}, a;}"
        : "=f"(r.x), "=f"(r.y) : "f"(a.x), "f"(a.y), "f"(b.x), "f"(b.y), "f"(-1.f));
    return r;
}

// the parts of two neighbouring elements, the first in the low half
__device__ __forceinline__ void thirds(float2 v, uint32_t &h, uint32_t &m, uint32_t &l) {
    auto first = [](float2 x) { return make_float2(__uint_as_float(__float_as_uint(x.x) & 0xffff0000u), __uint_as_float(__float_as_uint(x.y) & 0xffff0000u)); };
    auto pair = [](float2 x) { return __byte_perm(__float_as_uint(x.x), __float_as_uint(x.y), 0x7632); };
    h = pair(v);
    v = less_two(v, first(v));
    m = pair(v);
    v = less_two(v, first(v));
    l = pair(v);
}

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_bf16_from_zero(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// sum += the products of one run of 16 k: `w` the float4 of features g and g + 8 of MT tiles of 16 features, `a` that of row g of NT tiles
// of 8 rows, g = lane / 4; lane % 4 says which four k a float4 holds.
template <int MT, int NT> __device__ __forceinline__ void add_run(float (&sum)[MT][NT][4], const float4 (&w)[MT][2], const float4 (&a)[NT]) {
    constexpr int H = 0, M = 1, L = 2;
    uint32_t wp[3][MT][4], ap[3][NT][2];
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            thirds(make_float2(w[i][r].x, w[i][r].y), wp[H][i][r], wp[M][i][r], wp[L][i][r]);
            thirds(make_float2(w[i][r].z, w[i][r].w), wp[H][i][2 + r], wp[M][i][2 + r], wp[L][i][2 + r]);
        }
#pragma unroll
    for (int j = 0; j < NT; ++j) {
        thirds(make_float2(a[j].x, a[j].y), ap[H][j][0], ap[M][j][0], ap[L][j][0]);
        thirds(make_float2(a[j].z, a[j].w), ap[H][j][1], ap[M][j][1], ap[L][j][1]);
    }
    constexpr int PW[8] = {L, M, L, H, M, M, H, H}, PA[8] = {M, L, H, L, M, H, M, H};
    float acc[MT][NT][4];
#pragma unroll
    for (int p = 0; p < 8; ++p) {
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (p == 0 || p == 7) mma_bf16_from_zero(acc[i][j], wp[PW[p]][i], ap[PA[p]][j]);
                else mma_bf16(acc[i][j], wp[PW[p]][i], ap[PA[p]][j]);
            }
        if (p < 6) continue;
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j)
#pragma unroll
                for (int e = 0; e < 4; e += 2) {
                    const float2 v = add_two(make_float2(sum[i][j][e], sum[i][j][e + 1]), make_float2(acc[i][j][e], acc[i][j][e + 1]));
                    sum[i][j][e] = v.x, sum[i][j][e + 1] = v.y;
                }
    }
}
