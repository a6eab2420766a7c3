// Pairs of 32-bit multiply-adds (sm_100's packed form), and the product of two tiles in shared memory out of them.
#pragma once

#include "common.cuh"

// d = a * b + c on both halves, each rounded as the scalar instruction rounds.
__device__ __forceinline__ float2 fma2(float2 a, float2 b, float2 c) {
    float2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)),
          "l"(reinterpret_cast<unsigned long long&>(c)));
    return d;
}
__device__ __forceinline__ float2 mul2(float2 a, float2 b) {
    float2 d;
    asm("mul.rn.f32x2 %0, %1, %2;"
        : "=l"(reinterpret_cast<unsigned long long&>(d))
        : "l"(reinterpret_cast<unsigned long long&>(a)), "l"(reinterpret_cast<unsigned long long&>(b)));
    return d;
}

// acc[i][j] += sum over k < K of a[i lda + k] b[16 j ldb + k], the even and the odd k in a half each (K a multiple of 4): both
// operands as rows along k, 16 bytes for four steps of it, so that 8 shared loads feed 64 multiply-adds.
template <int UNROLL>
__device__ __forceinline__ void tile_product(const float* a, int lda, const float* b, int ldb, int K, float2 (&acc)[4][4]) {
#pragma unroll UNROLL
    for (int k = 0; k < K; k += 4) {
        float4 av[4], bv[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) av[i] = *reinterpret_cast<const float4*>(a + i * lda + k);
#pragma unroll
        for (int j = 0; j < 4; ++j) bv[j] = *reinterpret_cast<const float4*>(b + 16 * j * ldb + k);
#pragma unroll
        for (int i = 0; i < 4; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                acc[i][j] = fma2(make_float2(av[i].x, av[i].y), make_float2(bv[j].x, bv[j].y), acc[i][j]);
                acc[i][j] = fma2(make_float2(av[i].z, av[i].w), make_float2(bv[j].z, bv[j].w), acc[i][j]);
            }
    }
}
