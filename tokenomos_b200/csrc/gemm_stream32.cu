// Few-row matrix product of the true 32-bit path: out[M, N] = x[M, K] . W[N, K]^T (+ bias), M <= 8, all
// operands float32, 32-bit FMA sums on the CUDA cores.
//
// Such a product is bound by the stream of weight bytes (eight multiply-adds a weight at most, 128 lanes an SM:
// a third of what the cores can do at the copy bandwidth), so the split is the one that reads every weight row in
// whole 128-byte lines with many loads in flight: a CTA owns 2 to 8 weight rows and all of K, its 8 warps take alternate
// 128-wide slices of K, a lane 4 neighbouring columns of all rows, one to four slices asked for together (launch_stream32). The activations
// (64 KB at most for 8 rows of 2,048) are read the same way through L1. A lane then holds 4 x M partial sums; the
// warp adds them up with a halving exchange (31 shuffles for 32 sums instead of 160), the warps through shared memory.
// SWIGLU: the rows of W are all gate rows, then all up rows; the CTA takes as many channels of both and writes
// silu(gate) * up, so a decoded token needs no activation kernel.
//
// The kernel this replaces up to 8 rows (a 64 x 64 tile of gemm_simt.cu) filled its tile with rows that do not exist
// and ran N / 64 CTAs: the feed-forward of 1,024 x 4,608 at one row took 416 us in three launches, with this kernel
// 13.7 us in two (4.1 TB/s of weights).
#include "common.cuh"

namespace {

constexpr int S32_WARPS = 8, S32_SLICE = 128;

__device__ __forceinline__ float4 ld_weights(const float* p) {
    float4 v;
    asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];\n"
                 : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
                 : "l"(p));
    return v;
}

// Sums v[0 .. V) over the warp, V a power of two up to 32: lane l returns the total of v[l % V].
template <int V>
__device__ __forceinline__ float halving_sum(float (&v)[V], int lane) {
#pragma unroll
    for (int half = V / 2; half >= 1; half /= 2) {
        const bool upper = lane & half;
#pragma unroll
        for (int i = 0; i < half; ++i) {
            const float mine = upper ? v[i + half] : v[i], theirs = upper ? v[i] : v[i + half];
            v[i] = mine + __shfl_xor_sync(0xffffffffu, theirs, half);
        }
    }
    float s = v[0];
#pragma unroll
    for (int o = V; o < 32; o *= 2) s += __shfl_xor_sync(0xffffffffu, s, o);
    return s;
}

// ROWS weight rows a CTA, UNROLL slices of K a warp asked for together (see launch_stream32)
template <int MT, bool SWIGLU, int ROWS, int UNROLL>
__global__ void __launch_bounds__(S32_WARPS * 32, MT >= 4 && ROWS == 4 && UNROLL == 1 ? 4 : 0)
gemm_stream32_kernel(const float* x, int64_t ldx, const float* __restrict__ w, int64_t ldw,
                     const float* __restrict__ bias, float* out, int64_t ldo, int M, int N, int K) {
    constexpr int V = ROWS * MT;
    __shared__ float red[S32_WARPS][V];
    pdl_launch_dependents();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    // the CTA's rows of W: neighbours, or half as many gate rows and the up rows of the same channels
    const int channels = SWIGLU ? N / 2 : N;
    constexpr int OWN = SWIGLU ? ROWS / 2 : ROWS;
    const int c0 = blockIdx.x * OWN;
    const float* wr[ROWS];
    int row[ROWS];
#pragma unroll
    for (int r = 0; r < ROWS; ++r) {
        const int c = c0 + r % OWN;
        row[r] = min(c, channels - 1) + (r / OWN) * channels;       // (a row past the end repeats the last one)
        wr[r] = w + (size_t)row[r] * ldw;
    }
    float acc[V];
#pragma unroll
    for (int i = 0; i < V; ++i) acc[i] = 0.f;
    const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
    bool waited = false;
    for (int k0 = warp * S32_SLICE; k0 < K; k0 += S32_WARPS * S32_SLICE * UNROLL) {
        float4 wv[UNROLL][ROWS];
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int k = k0 + u * S32_WARPS * S32_SLICE + lane * 4;
#pragma unroll
            for (int r = 0; r < ROWS; ++r) wv[u][r] = k < K ? ld_weights(wr[r] + k) : zero;
        }
        if (!waited) {                    // the weights are no kernel's output, the activations are
            pdl_wait();
            waited = true;
        }
#pragma unroll
        for (int u = 0; u < UNROLL; ++u) {
            const int k = k0 + u * S32_WARPS * S32_SLICE + lane * 4;
            if (k >= K) continue;         // (zero weights would turn an infinite activation into NaN)
#pragma unroll
            for (int m = 0; m < MT; ++m) {
                if (m >= M) break;
                const float4 xv = *reinterpret_cast<const float4*>(x + (size_t)m * ldx + k);
#pragma unroll
                for (int r = 0; r < ROWS; ++r) {
                    float a = acc[r * MT + m];
                    a = fmaf(wv[u][r].x, xv.x, a);
                    a = fmaf(wv[u][r].y, xv.y, a);
                    a = fmaf(wv[u][r].z, xv.z, a);
                    acc[r * MT + m] = fmaf(wv[u][r].w, xv.w, a);
                }
            }
        }
    }
    if (!waited) pdl_wait();
    const float total = halving_sum<V>(acc, lane);
    if (lane < V) red[warp][lane] = total;
    __syncthreads();
    const int r = threadIdx.x / MT, m = threadIdx.x % MT;
    if (r < OWN && m < M && c0 + r < channels) {
        float sum = 0.f, up = 0.f;
#pragma unroll
        for (int wv = 0; wv < S32_WARPS; ++wv) {
            sum += red[wv][r * MT + m];
            if (SWIGLU) up += red[wv][(r + OWN) % ROWS * MT + m];
        }
        if (bias != nullptr) {
            sum += bias[c0 + r];
            if (SWIGLU) up += bias[channels + c0 + r];
        }
        out[(size_t)m * ldo + c0 + r] = SWIGLU ? silu_as<float>(sum) * up : sum;
    }
}

// 4 rows a CTA and two slices a warp in flight, but:
// - up to 1,024 columns (one slice a warp) 8 rows for one to four tokens, one wave of CTAs instead of two (us at 9,216 x 1,024, SwiGLU:
//   one token 7.0, with 4 rows 9.3, two 7.8 and 8.4, four 10.9 and 11.4; two tokens from 8,192 rows on, four from 4,096);
// - one token beyond 2,048 columns four slices (4,096 x 4,096 11.7 and 13.1), and 2 rows a CTA where the matrix has few (1,024 x 4,608
//   3.8 and 4.9, 2,048 x 10,752 14.0 and 16.4; two tokens and more are slower that way, 2,048 x 8,192 15.5 and 11.8);
// - more than two tokens one slice, whose registers let four CTAs share an SM instead of two (three with four tokens), where the
//   matrix has more rows than those hold at once (eight tokens: 2,048 x 8,192 21.1 and 31.4, 16,384 x 2,048 36.3 and 44.2, 9,216 x
//   1,024 13.5 and 18.9, 1,024 x 4,608 12.3 and 10.5; four: 2,048 x 8,192 13.7 and 20.6), with four tokens and up to 2,048 columns only
//   while four CTAs an SM are all there are (2,048 x 2,048 4.3 and 6.5, 3,072 x 2,048 7.8 and 7.1).
template <bool SWIGLU>
void launch_stream32(const float* x, int64_t ldx, const float* w, int64_t ldw, const float* bias, float* out, int64_t ldo,
                     int M, int N, int K, cudaStream_t stream) {
#define TK_S32(MT, ROWS, UNROLL)                                                                                              \
    tk_launch(gemm_stream32_kernel<MT, SWIGLU, ROWS, UNROLL>, dim3(ceil_div(SWIGLU ? N / 2 : N, SWIGLU ? ROWS / 2 : ROWS)),   \
              dim3(S32_WARPS * 32), 0, stream, x, ldx, w, ldw, bias, out, ldo, M, N, K)
    const int once = S32_WARPS * S32_SLICE, wave = 4 * 148;          // columns of one slice a warp; rows of a CTA an SM
#define TK_S32_K(MT)                                                                                              \
    do {                                                                                                          \
        if (MT <= 4 && K <= once && N >= (MT == 1 ? 0 : MT == 2 ? 8192 : 4096)) TK_S32(MT, (MT <= 4 ? 8 : 4), 1); \
        else if (MT == 1 && K > 2 * once && N <= 2048) TK_S32(MT, (MT == 1 ? 2 : 4), (MT == 1 ? 4 : 2));          \
        else if (MT == 1 && K > 2 * once) TK_S32(MT, 4, (MT == 1 ? 4 : 2));                                       \
        else if ((MT == 8 && N > 2 * wave) || (MT == 4 && K > once && N > 3 * wave && (K > 2 * once || N <= 4 * wave))) \
            TK_S32(MT, 4, (MT >= 4 ? 1 : 2));                                                                     \
        else TK_S32(MT, 4, 2);                                                                                    \
    } while (0)
    if (M == 1) TK_S32_K(1);
    else if (M == 2) TK_S32_K(2);
    else if (M <= 4) TK_S32_K(4);
    else TK_S32_K(8);
#undef TK_S32_K
#undef TK_S32
}

}  // namespace

TK_API int tk_gemm_stream32_max_rows() { return 8; }

// x: float32 [M, K] rows ldx apart, w: float32 [N, K] rows ldw apart (16-byte aligned rows, K a multiple of 4);
// out: [M, N], or [M, N / 2] with swiglu.
TK_API int tk_gemm_stream32(const void* x, int64_t ldx, const void* w, int64_t ldw, const float* bias, void* out, int64_t ldo,
                            int M, int N, int K, int swiglu, cudaStream_t stream) {
    TK_CHECK_ARG(M > 0 && M <= tk_gemm_stream32_max_rows() && N > 0 && K > 0, "gemm_stream32: M=%d (1..%d) N=%d K=%d", M,
                 tk_gemm_stream32_max_rows(), N, K);
    TK_CHECK_ARG(K % 4 == 0 && ldx % 4 == 0 && ldw % 4 == 0 && (uintptr_t)x % 16 == 0 && (uintptr_t)w % 16 == 0,
                 "gemm_stream32: K and the leading dimensions must be multiples of 4, bases 16-byte aligned");
    TK_CHECK_ARG((M == 1 || ldx >= K) && ldw >= K && (!swiglu || N % 2 == 0) && ldo >= (swiglu ? N / 2 : N),
                 "gemm_stream32: leading dimensions too small, or %d rows of gate and up", N);
    if (swiglu) launch_stream32<true>((const float*)x, ldx, (const float*)w, ldw, bias, (float*)out, ldo, M, N, K, stream);
    else launch_stream32<false>((const float*)x, ldx, (const float*)w, ldw, bias, (float*)out, ldo, M, N, K, stream);
    TK_CHECK_LAUNCH("gemm_stream32");
    return 0;
}
