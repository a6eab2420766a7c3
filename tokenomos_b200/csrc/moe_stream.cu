// The grouped product of a mixture of experts for steps of a few tokens: C[m, :] = act(A[row(m), :] . W[g]^T) with g the
// expert of m's tile, bfloat16, 32-bit sums on the tensor cores (mma.sync m16n8k16, weight rows on the M axis).
//
// With a few rows an expert such a step is a stream of the chosen experts' weights and nothing else, so a CTA owns 16
// weight rows of one expert and all of K, its 8 warps take alternate 64-wide slices, every thread reads its share of the rows
// with 16-byte loads straight into registers (whole 128-byte lines, two slices in flight) and the tile's 8 or 16 input rows
// the same way through L1: gemm_skinny.cu's form, with the rows gathered and an expert picked by the tile. The tiles of
// 64 rows this replaces here staged 64 input rows, nearly all of them padding, for every 64 or 128 weight rows, through
// shared memory and one barrier every 32 columns. A mixture of 32 experts of 2,048 x 1,536 at 16 tokens of 4 experts each:
// 132 us with the shared expert and the routing around it (4.2 TB/s over all), 215 before.
#include "common.cuh"

namespace {

constexpr int MS_WARPS = 8, MS_ROWS = 16, MS_SLICE = 64, MS_UNROLL = 2;

__device__ __forceinline__ void ms_mma(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                       uint32_t b1) {
    asm volatile(
        "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
        : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint4 ms_weights(const void* p) {
    uint4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];\n" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "l"(p));
    return v;
}

// TILE: rows of a tile (8 or 16). row_token[m] < 0: a row of padding, neither read nor written; gather: m reads row row_token[m]
// of A, else row m. act 0: none; 1: relu(v)^2; 2 and 3: the weight's rows are gates and ups alternating in runs of 8, C has
// N / 2 columns (2: silu(gate) * up; 3: g = min(gate, limit), u = clamp(up, -limit, limit), limit <= 0 no clamp, g
// sigmoid(alpha g) (u + shift)), gate and up rounded first, as a product that is stored would be.
template <int TILE>
__global__ void __launch_bounds__(MS_WARPS * 32)
moe_stream_kernel(const __nv_bfloat16* A, int64_t lda, const int* row_token, int gather, const __nv_bfloat16* __restrict__ W,
                  const int* tile_group, __nv_bfloat16* C, int64_t ldc, int N, int K, int act, float limit, float alpha,
                  float shift) {
    constexpr int TG = TILE / 8;
    __shared__ float red[MS_WARPS][MS_ROWS][TILE];
    pdl_launch_dependents();
    pdl_wait();
    const int expert = tile_group[blockIdx.y];
    if (expert < 0) return;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    const int n0 = blockIdx.x * MS_ROWS, m0 = blockIdx.y * TILE;
    const __nv_bfloat16* w = W + (size_t)expert * N * K;
    const bool ok0 = n0 + g < N, ok1 = n0 + g + 8 < N;
    const __nv_bfloat16 *w0 = w + (size_t)(ok0 ? n0 + g : 0) * K, *w1 = w + (size_t)(ok1 ? n0 + g + 8 : 0) * K;
    const __nv_bfloat16* xr[TG];
    bool x_ok[TG];
#pragma unroll
    for (int i = 0; i < TG; ++i) {
        const int m = m0 + 8 * i + g, tok = row_token[m];
        x_ok[i] = tok >= 0;
        xr[i] = A + (size_t)(x_ok[i] ? (gather ? tok : m) : 0) * lda;
    }
    float acc[TG][4];
#pragma unroll
    for (int i = 0; i < TG; ++i)
#pragma unroll
        for (int e = 0; e < 4; ++e) acc[i][e] = 0.f;
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const int slices = (K + MS_SLICE - 1) / MS_SLICE;
    for (int s0 = warp; s0 < slices; s0 += MS_WARPS * MS_UNROLL) {
        uint4 wa[MS_UNROLL][2], wb[MS_UNROLL][2];
#pragma unroll
        for (int u = 0; u < MS_UNROLL; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = s0 + u * MS_WARPS, k = s * MS_SLICE + h * 32 + 8 * t;
                const bool in = s < slices && k < K;
                wa[u][h] = in && ok0 ? ms_weights(w0 + k) : zero;
                wb[u][h] = in && ok1 ? ms_weights(w1 + k) : zero;
            }
#pragma unroll
        for (int u = 0; u < MS_UNROLL; ++u)
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int s = s0 + u * MS_WARPS, k = s * MS_SLICE + h * 32 + 8 * t;
                const bool in = s < slices && k < K;
#pragma unroll
                for (int i = 0; i < TG; ++i) {
                    const uint4 x = in && x_ok[i] ? *reinterpret_cast<const uint4*>(xr[i] + k) : zero;
                    // (the K index of a register pair is permuted alike for both operands: one 16-byte load feeds two steps)
                    ms_mma(acc[i], wa[u][h].x, wb[u][h].x, wa[u][h].y, wb[u][h].y, x.x, x.y);
                    ms_mma(acc[i], wa[u][h].z, wb[u][h].z, wa[u][h].w, wb[u][h].w, x.z, x.w);
                }
            }
    }
    // acc[i]: weight rows g and g + 8, input rows 8 i + 2 t and + 1
#pragma unroll
    for (int i = 0; i < TG; ++i) {
        *reinterpret_cast<float2*>(&red[warp][g][8 * i + 2 * t]) = make_float2(acc[i][0], acc[i][1]);
        *reinterpret_cast<float2*>(&red[warp][g + 8][8 * i + 2 * t]) = make_float2(acc[i][2], acc[i][3]);
    }
    __syncthreads();
    const int per = act >= 2 ? 8 : MS_ROWS;
    for (int i = threadIdx.x; i < per * TILE; i += MS_WARPS * 32) {
        const int r = i % per, m = i / per;                   // columns fastest: neighbours in memory
        if (row_token[m0 + m] < 0 || n0 + r + (act >= 2 ? 8 : 0) >= N) continue;
        float v = 0.f, up = 0.f;
#pragma unroll
        for (int wv = 0; wv < MS_WARPS; ++wv) {
            v += red[wv][r][m];
            if (act >= 2) up += red[wv][r + 8][m];
        }
        if (act >= 2) {
            float a = round_as<__nv_bfloat16>(v), u = round_as<__nv_bfloat16>(up);
            if (act == 3) {
                if (limit > 0.f) {
                    a = fminf(a, limit);
                    u = fminf(fmaxf(u, -limit), limit);
                }
                v = a / (1.f + expf(-alpha * a)) * (u + shift);
            } else {
                v = a / (1.f + expf(-a)) * u;
            }
            C[(size_t)(m0 + m) * ldc + n0 / 2 + r] = __float2bfloat16_rn(v);
        } else {
            if (act == 1) {
                v = fmaxf(v, 0.f);
                v *= v;
            }
            C[(size_t)(m0 + m) * ldc + n0 + r] = __float2bfloat16_rn(v);
        }
    }
}

}  // namespace

// A: bfloat16 rows lda apart; row_token: int32 [rows]; W: [experts, N, K]; tile_group: int32 [rows / tile] (-1: unused);
// C: [rows, N], or [rows, N / 2] with a gated activation. rows: whole tiles of 8 or 16.
TK_API int tk_moe_stream(const void* A, int64_t lda, const int* row_token, int gather, const void* W, const int* tile_group,
                         void* C, int64_t ldc, int rows, int N, int K, int act, int tile, float limit, float alpha, float shift,
                         cudaStream_t stream) {
    TK_CHECK_ARG((tile == 8 || tile == 16) && rows >= 0 && rows % tile == 0 && rows / tile <= 65535 && N > 0 && K > 0,
                 "moe_stream: %d rows in tiles of %d, N=%d K=%d", rows, tile, N, K);
    TK_CHECK_ARG(K % 8 == 0 && lda % 8 == 0 && (uintptr_t)A % 16 == 0 && (uintptr_t)W % 16 == 0 && row_token != nullptr,
                 "moe_stream: rows in whole 16-byte chunks");
    TK_CHECK_ARG(act >= 0 && act <= 3 && (act < 2 || N % 16 == 0), "moe_stream: activation %d with %d columns", act, N);
    if (rows == 0) return 0;
    const dim3 grid(ceil_div(N, MS_ROWS), rows / tile), block(MS_WARPS * 32);
    auto a = (const __nv_bfloat16*)A;
    auto w = (const __nv_bfloat16*)W;
    auto c = (__nv_bfloat16*)C;
    if (tile == 8)
        tk_launch(moe_stream_kernel<8>, grid, block, 0, stream, a, lda, row_token, gather, w, tile_group, c, ldc, N, K, act, limit,
                  alpha, shift);
    else
        tk_launch(moe_stream_kernel<16>, grid, block, 0, stream, a, lda, row_token, gather, w, tile_group, c, ldc, N, K, act, limit,
                  alpha, shift);
    TK_CHECK_LAUNCH("moe_stream");
    return 0;
}
