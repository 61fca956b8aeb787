// float32 products on the tensor cores, both operands in two tf32 halves: w = hi + lo, hi being w rounded to the 11 bits of a tf32 number
// and lo what that lost (exact; the tensor core reads its first 11 bits).  The products lo hi, hi lo and then hi hi of a run of 16 k are
// added up by mma.sync (m16n8k8) from zero and the run's sum joins the caller's in float32.  The tensor core cuts what it adds instead of
// rounding it, which is why so little is added up there (K = 1024 in one go, random signs: 2.5e-6 off 64 bits; run by run
// 1.3e-7, a chain of FMAs 5.8e-7); what hi lo and lo hi lose is under 2^-11 of that.
#pragma once
#include <stdint.h>

__device__ __forceinline__ void split(float x, uint32_t &hi, uint32_t &lo) {
    hi = (__float_as_uint(x) + 0x1000u) & 0xffffe000u;
    lo = __float_as_uint(x - __uint_as_float(hi));
}
__device__ __forceinline__ void mma_tf32(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
__device__ __forceinline__ void mma_tf32_from_zero(float (&c)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k8.row.col.f32.tf32.tf32.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
        : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(0.f));
}

// sum += the products of one run of 16 k: `w` the float4 of features g and g + 8 of MT tiles of 16 features, `a` that of row g of NT tiles
// of 8 rows, g = lane / 4; lane % 4 says which four k a float4 holds.
template <int MT, int NT> __device__ __forceinline__ void add_run(float (&sum)[MT][NT][4], const float4 (&w)[MT][2], const float4 (&a)[NT]) {
    float acc[MT][NT][4];
    uint32_t wh[2][MT][4], ah[2][NT][2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {           // two of every lane's four k at a time
        uint32_t wl[MT][4], al[NT][2];
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                split(h ? w[i][r].z : w[i][r].x, wh[h][i][r], wl[i][r]);
                split(h ? w[i][r].w : w[i][r].y, wh[h][i][2 + r], wl[i][2 + r]);
            }
#pragma unroll
        for (int j = 0; j < NT; ++j) {
            split(h ? a[j].z : a[j].x, ah[h][j][0], al[j][0]);
            split(h ? a[j].w : a[j].y, ah[h][j][1], al[j][1]);
        }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) {
                if (h == 0) mma_tf32_from_zero(acc[i][j], wl[i], ah[h][j]);
                else mma_tf32(acc[i][j], wl[i], ah[h][j]);
            }
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) mma_tf32(acc[i][j], wh[h][i], al[j]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < MT; ++i)
#pragma unroll
            for (int j = 0; j < NT; ++j) mma_tf32(acc[i][j], wh[h][i], ah[h][j]);
#pragma unroll
    for (int i = 0; i < MT; ++i)
#pragma unroll
        for (int j = 0; j < NT; ++j)
#pragma unroll
            for (int e = 0; e < 4; ++e) sum[i][j][e] += acc[i][j][e];
}
