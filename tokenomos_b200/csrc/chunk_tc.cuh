// Chunks of 64 tokens on the 16-bit tensor cores with 32-bit arithmetic: what the recurrences that go chunk by chunk share. A chunk's
// 64 x 64 matrices (row t, column s <= t) lie in memory as three 16-bit parts, each as shared memory holds it (128-byte rows,
// swizzled); operands go from warp to warp as registers hold them ([..][lane] 16 bytes).
//
// Chunks count from each sequence's first token of the step; sequence s has the slots cu_seqlens[s] / 64 + s and up.
#pragma once

#include <math.h>

#include "packed.cuh"
#include "paged_tiles.cuh"
#include "parts.cuh"

namespace {

constexpr int DC_T = 64;                       // tokens of a chunk
constexpr int DC_LD = DC_T + 4;                // row of a 64 x 64 matrix of floats in shared memory
constexpr int DC_PART = DC_T * DC_T * 2;       // bytes of one 16-bit part of such a matrix

__device__ __forceinline__ uint32_t shared_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

struct Chunk64 {
    int first, nt;                             // the chunk's first token in the step and its count (not above 0: no such chunk)
};
__device__ __forceinline__ Chunk64 chunk_of(const int* cu_seqlens, int n_seqs, int slot) {
    // the last sequence whose first slot is not past this one (every warp looks for itself, 32 sequences at a time)
    int s = -1;
    for (int s0 = 0; s0 < n_seqs; s0 += 32) {
        const int i = s0 + (threadIdx.x & 31);
        const unsigned before = __ballot_sync(0xffffffffu, i < n_seqs && cu_seqlens[i] / DC_T + i <= slot);
        s += __popc(before);
        if (before != 0xffffffffu) break;
    }
    const int begin = cu_seqlens[s], len = cu_seqlens[s + 1] - begin, j = slot - (begin / DC_T + s);
    return {begin + j * DC_T, min(DC_T, len - j * DC_T)};
}

// The n-th of the ten blocks of 16 x 16 on and left of the diagonal of (rows of `left`) (rows of `right`)^T, both tiles of 64 x D;
// by one warp, into a matrix of floats in shared memory.
template <int D>
__device__ __forceinline__ void lower_block(float* mat, uint32_t left, uint32_t right, int n, int lane) {
    const int bi = n < 1 ? 0 : n < 3 ? 1 : n < 6 ? 2 : 3, bj = n - bi * (bi + 1) / 2;
    float c[2][2][4];                          // (even and odd steps apart: half the sums that are cut off)
#pragma unroll
    for (int e = 0; e < 16; ++e) c[e >> 3][(e >> 2) & 1][e & 3] = 0.f;
#pragma unroll
    for (int ks = 0; ks < D / 16; ++ks) {
        uint32_t a[4], b[4];
        ldmatrix_x4(a, left + tile_off<D>(bi * 16 + (lane & 15), ks * 2 + (lane >> 4)));
        ldmatrix_x4(b, right + tile_off<D>(bj * 16 + (lane & 7) + (lane >> 4) * 8, ks * 2 + ((lane >> 3) & 1)));
        mma16816(c[ks & 1][0], a, b[0], b[1]);
        mma16816(c[ks & 1][1], a, b[2], b[3]);
    }
    float* out = mat + (bi * 16 + (lane >> 2)) * DC_LD + bj * 16 + 2 * (lane & 3);
#pragma unroll
    for (int t8 = 0; t8 < 2; ++t8) {
        *reinterpret_cast<float2*>(out + t8 * 8) = make_float2(c[0][t8][0] + c[1][t8][0], c[0][t8][1] + c[1][t8][1]);
        *reinterpret_cast<float2*>(out + 8 * DC_LD + t8 * 8) = make_float2(c[0][t8][2] + c[1][t8][2], c[0][t8][3] + c[1][t8][3]);
    }
}

// Row and first column of a lane's pair of neighbouring columns in the n-th of a warp's steps over the blocks of 16 x 16 on and left
// of the diagonal, four warps sharing them: four rows a step in the first 16, two in the next, then one (in rows 32 to 47 the last
// lanes have none: column 64).
constexpr int DC_STEPS = 1 + 2 + 4 + 4;
__device__ __forceinline__ int2 triangle_step(int n, int warp, int lane) {
    if (n < 1) return make_int2(4 * warp + (lane >> 3), 2 * (lane & 7));
    if (n < 3) return make_int2(16 + 8 * (n - 1) + 2 * warp + (lane >> 4), 2 * (lane & 15));
    return make_int2(32 + 4 * (n - 3) + warp, n < 7 && lane >= 24 ? DC_T : 2 * lane);
}
__device__ __forceinline__ void store_parts(uint8_t* part, int2 at, float a, float b) {
    uint32_t hi, mi, lo;
    take_apart(a, b, hi, mi, lo);
    uint8_t* dst = part + tile_off<DC_T>(at.x, at.y >> 3) + (at.y & 6) * 2;
    *reinterpret_cast<uint32_t*>(dst) = hi;
    *reinterpret_cast<uint32_t*>(dst + DC_PART) = mi;
    *reinterpret_cast<uint32_t*>(dst + 2 * DC_PART) = lo;
}

__device__ __forceinline__ void dc_cut(uint32_t (&a)[3][4], const float (&c0)[4], const float (&c1)[4]) {
    cut_apart(c0[0], c0[1], a[0][0], a[1][0], a[2][0]);
    cut_apart(c0[2], c0[3], a[0][1], a[1][1], a[2][1]);
    cut_apart(c1[0], c1[1], a[0][2], a[1][2], a[2][2]);
    cut_apart(c1[2], c1[3], a[0][3], a[1][3], a[2][3]);
}

__device__ __forceinline__ void dc_sync() { asm volatile("bar.sync 0;" ::: "memory"); }
__device__ __forceinline__ void dc_give(uint8_t* at, const uint32_t (&a)[3][4]) {
#pragma unroll
    for (int p = 0; p < 3; ++p) *reinterpret_cast<uint4*>(at + p * 512) = make_uint4(a[p][0], a[p][1], a[p][2], a[p][3]);
}
__device__ __forceinline__ void dc_take(uint32_t (&a)[3][4], const uint8_t* at) {
#pragma unroll
    for (int p = 0; p < 3; ++p) {
        const uint4 v = *reinterpret_cast<const uint4*>(at + p * 512);
        a[p][0] = v.x, a[p][1] = v.y, a[p][2] = v.z, a[p][3] = v.w;
    }
}
template <int N>
__device__ __forceinline__ void dc_zero(float (&c)[N][4]) {
#pragma unroll
    for (int n = 0; n < N; ++n)
#pragma unroll
        for (int e = 0; e < 4; ++e) c[n][e] = 0.f;
}
// (high, rest) of two neighbouring tiles += a float's three parts times a 16-bit operand
__device__ __forceinline__ void dc_three(float (&hi0)[4], float (&hi1)[4], float (&lo0)[4], float (&lo1)[4], const uint32_t (&a)[3][4],
                                         const uint32_t (&b)[4]) {
    mma16816(lo0, a[2], b[0], b[1]);
    mma16816(lo1, a[2], b[2], b[3]);
    mma16816(hi0, a[0], b[0], b[1]);
    mma16816(hi1, a[0], b[2], b[3]);
    mma16816(lo0, a[1], b[0], b[1]);
    mma16816(lo1, a[1], b[2], b[3]);
}

}  // namespace
